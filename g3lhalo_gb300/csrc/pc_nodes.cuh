// pc_nodes.cuh -- how the precompute's warps share the nodes of one bisection tree.
//
// A slot of the node table is claimed by compare-and-swap, filled, and published with a
// release store; a node may be read only by a thread whose view is ordered behind that
// store.  The protocol is written over a Table, so that a host test can run it against one
// that keeps track of this order (the device's loads happen to keep it anyway, so results
// do not show a step that is missing).
#pragma once

namespace g3l {

enum : unsigned { NODE_FREE = 0, NODE_FILLING = 1, NODE_READY = 2 };
constexpr int PC_PROBES = 16;

// Find a node from slot ix on (mask + 1 slots).  Table: acquire(ix), the slot's state by an
// acquire load; claim(ix), compare-and-swap of FREE by FILLING, which returns the old state
// and orders nothing; match(ix), whether a ready slot holds the node.  mode 2: ready at the
// returned slot, 1: claimed by this caller (to be filled and published), 0: evaluate the
// node without the table.
#pragma nv_exec_check_disable
template <class Table>
__host__ __device__ __forceinline__ int node_find(Table &C, unsigned ix, unsigned mask, int &mode)
{
    for (int p = 0; p < PC_PROBES; ++p, ix = (ix + 1) & mask) {
        unsigned st = C.acquire((int)ix);
        if (st == NODE_FREE) {
            st = C.claim((int)ix);
            if (st == NODE_FREE) {
                mode = 1;
                return (int)ix;
            }
            st = C.acquire((int)ix);  // the claim orders nothing: the slot may be ready by now
        }
        if (st == NODE_FILLING) break;  // perhaps by this node's first visitor
        if (C.match((int)ix)) {
            mode = 2;
            return (int)ix;
        }
    }
    mode = 0;
    return -1;
}

// Lane 0 of a half-warp has looked a node up; its other lanes take over the finding (every
// lane of the warp calls).  Lanes: bcast(v), lane 0's v; sync(), a barrier of the warp that
// orders memory.
#pragma nv_exec_check_disable
template <class Lanes>
__host__ __device__ __forceinline__ void node_share(const Lanes &L, int &mode, int &ix)
{
    mode = L.bcast(mode);
    ix = L.bcast(ix);
    L.sync();  // lane 0's acquire load then comes before every lane's reads of the node
}

}  // namespace g3l
