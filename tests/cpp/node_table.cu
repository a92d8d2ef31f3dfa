// The node table's protocol (pc_nodes.cuh) on the host, over a table that keeps track of
// which reads are ordered behind a node's publication.  Prints the first failure and exits
// 1, or prints "ok" and exits 0.
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>

#include <pthread.h>

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

// A warp of 32 threads.  seen[lane]: the slots whose publication the lane's reads are ordered
// behind, a bit each; a broadcast moves a value and orders nothing, a barrier makes what any
// lane is ordered behind hold for all.
struct Warp {
    pthread_barrier_t bar;
    int val[32];
    unsigned seen[32] = {};
    Warp() { pthread_barrier_init(&bar, nullptr, 32); }
    ~Warp() { pthread_barrier_destroy(&bar); }
    void wait() { pthread_barrier_wait(&bar); }
};
struct Lanes {
    Warp &w;
    int lane;
    int bcast(int v) const
    {
        w.val[lane] = v;
        w.wait();
        const int r = w.val[lane & 16];
        w.wait();
        return r;
    }
    void sync() const
    {
        unsigned all = 0;
        w.wait();
        for (unsigned s : w.seen) all |= s;
        w.wait();
        w.seen[lane] = all;
        w.wait();
    }
};
struct LaneTable {  // slots 3 and 9 are ready, the nodes of the first and the second half-warp
    Warp &w;
    int lane, want;
    unsigned acquire(int ix) const
    {
        w.seen[lane] |= 1u << ix;
        return NODE_READY;
    }
    unsigned claim(int) const { return NODE_READY; }
    bool match(int ix) const { return ix == want; }
};

static void warp_reads_nodes()
{
    Warp w;
    std::vector<std::thread> lanes;
    bool ordered[32];
    int slot[32], modes[32];
    for (int lane = 0; lane < 32; ++lane)
        lanes.emplace_back([&, lane] {
            const LaneTable T{w, lane, lane < 16 ? 3 : 9};
            int mode = 0, ix = -1;
            if ((lane & 15) == 0) ix = node_find(T, 2, 31, mode);
            node_share(Lanes{w, lane}, mode, ix);
            slot[lane] = ix;
            modes[lane] = mode;
            ordered[lane] = ix >= 0 && ((w.seen[lane] >> ix) & 1u);
        });
    for (auto &t : lanes) t.join();
    for (int lane = 0; lane < 32; ++lane) {
        check(modes[lane] == 2 && slot[lane] == (lane < 16 ? 3 : 9), "lanes take over lane 0's finding");
        check(ordered[lane], "a lane reads a node that only lane 0 is ordered behind");
    }
}

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
    warp_reads_nodes();
    std::printf("ok\n");
    return 0;
}
