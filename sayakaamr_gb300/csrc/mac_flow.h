// The smoothing phase of one tower as one cooperative launch (mac_flow.cu).
#pragma once

#include "mac_device.h"

namespace sayaka_gb300 {

// tags of one launch: a cell's number of updates, at most kFlowTags - 2
constexpr unsigned kFlowTags = 32;
// tries of a wait before it gives up: about half a second
constexpr int kFlowPolls = 1 << 20;

// blocks that one launch can hold (0: blocks of another kind)
int flow_capacity(const Topo &t);
// words of the edge exchange, zeroed once; epoch: two zeroed words
size_t flow_words(const Topo &t);
// Tower of parity groups A and B (with halo descriptors): the prolongation of
// level `level` and nsweep red-black sweeps, launch_prolong_red's and
// launch_rbgs's values in their order.  grid: at least the groups' entries (of
// reduced lists: their active ones) and at most flow_capacity(t); nsweep <
// kFlowTags - 1.  alive: with reduced lists, the blocks they hold (else null).
// limit: tries of a wait.
cudaError_t launch_flow(const Topo &t, const Coef<float> &c, const BlockList &A, const BlockList &B, int level,
                        int nsweep, int grid, float *phi, const float *rhs, const int *guard,
                        unsigned long long *words, unsigned *epoch, const int *alive, cudaStream_t s,
                        int limit = kFlowPolls);

}  // namespace sayaka_gb300
