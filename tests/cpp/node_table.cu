// The node table's protocol (pc_nodes.cuh) on the host, over a table that keeps track of
// which reads are ordered behind a node's publication.  Prints the first failure and exits
// 1, or prints "ok" and exits 0.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "pc_nodes.cuh"

using namespace g3l;

static void check(bool ok, const char *what)
{
    if (ok) return;
    std::printf("failed: %s\n", what);
    std::exit(1);
}

// One thread's view of a table of 32 slots.  other: what another thread makes of a slot
// between this thread's load and its compare-and-swap (0 = nothing).
struct Table {
    std::vector<unsigned> state = std::vector<unsigned>(32, NODE_FREE), other = std::vector<unsigned>(32, 0u);
    std::vector<int> key = std::vector<int>(32, 0);
    std::vector<bool> ordered = std::vector<bool>(32, false);  // an acquire load saw it ready
    int want = 7, matches = 0;
    unsigned acquire(int ix)
    {
        if (state[ix] == NODE_READY) ordered[ix] = true;
        return state[ix];
    }
    unsigned claim(int ix)
    {
        if (other[ix]) state[ix] = other[ix];
        const unsigned old = state[ix];
        if (old == NODE_FREE) state[ix] = NODE_FILLING;
        return old;
    }
    bool match(int ix)
    {
        ++matches;
        check(state[ix] == NODE_READY, "key of a slot that is not ready is read");
        check(ordered[ix], "key read without an acquire load of the published state");
        return key[ix] == want;
    }
};

int main()
{
    int mode;
    {
        Table t;  // free: claimed
        check(node_find(t, 30, 31, mode) == 30 && mode == 1 && t.state[30] == NODE_FILLING, "free slot");
    }
    {
        Table t;  // ready, this node, behind another node and around the table's end
        t.state[31] = t.state[0] = NODE_READY;
        t.key[0] = 7;
        check(node_find(t, 31, 31, mode) == 0 && mode == 2, "ready slot");
    }
    {
        Table t;  // being filled
        t.state[5] = NODE_FILLING;
        check(node_find(t, 5, 31, mode) == -1 && mode == 0 && t.matches == 0, "slot being filled");
    }
    {
        Table t;  // claimed by another thread first, and not published yet
        t.other[5] = NODE_FILLING;
        check(node_find(t, 5, 31, mode) == -1 && mode == 0 && t.matches == 0, "lost claim");
    }
    {
        Table t;  // claimed and published by another thread in between
        t.other[5] = NODE_READY;
        t.key[5] = 7;
        check(node_find(t, 5, 31, mode) == 5 && mode == 2, "lost claim, published");
    }
    {
        Table t;  // the same with another node: the next slot is tried
        t.other[5] = NODE_READY;
        check(node_find(t, 5, 31, mode) == 6 && mode == 1, "lost claim, another node");
    }
    {
        Table t;  // a run of PC_PROBES other nodes
        for (int i = 0; i < PC_PROBES; ++i) t.state[i] = NODE_READY;
        check(node_find(t, 0, 31, mode) == -1 && mode == 0 && t.matches == PC_PROBES, "probe run exhausted");
    }
    std::printf("ok\n");
    return 0;
}
