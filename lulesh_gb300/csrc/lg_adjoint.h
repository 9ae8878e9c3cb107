// lg_adjoint.h -- the checkpointed adjoint's internal entry point (lg_adjoint.cu),
// called by the C ABI (lg_api.cu), which owns the handle.
#pragma once

#include <cuda_runtime.h>

#include <vector>

#include "lg_device.h"
#include "lg_kernelset.h"

namespace lg {

// The state fields the adjoint carries, in the order of its seed and
// gradient arrays: node x y z xd yd zd, element e p q v ss.
constexpr int kAdjFields = 11;

struct AdjointIO;

// What a handle keeps between calls: the limiter's reverse neighbour map on the
// device (drop_map when the topology changes) and the sweep's memory (kept: counted
// in the bound on what all handles keep).
struct AdjointWork {
    int *revStart = nullptr, *revEntry = nullptr;
    char *arena = nullptr;
    size_t held = 0;
    bool kept = false;
    int reverse_map(const AdjointIO &io, int E, cudaStream_t st);
    int reserve(size_t bytes, char **out);
    void release();   // after a sweep: keeps the arena within the bound
    void free_arena();
    void drop_map();
    void drop();
};

struct AdjointIO {
    const DevState *ds;
    const KernelSet *ks;
    cudaGraphExec_t cycle;      // one forward cycle
    cudaStream_t stream;
    Ctl *h_ctl;                 // pinned host copy of the control block
    const double *dts;          // host: frozen time steps of the cycles run
    int ncycles, ckpt_k;
    // the objective: either the masked terminal energy (mask non-null; E
    // entries) or the adjoint of the final state given field by field
    // (seed[f], host, NULL for zero)
    const unsigned char *mask;
    const double *const *seed;
    // host outputs: dJ / d(initial field f), NULL when not wanted (with a
    // mask, grad[6] receives dJ/de)
    double *const *grad;
    double hgcoef;
    AdjointWork *work;
    const std::vector<int> *lxim, *lxip, *letam, *letap, *lzetam, *lzetap, *elemBC;
};

// Runs the forward cycles with checkpoints, then the reverse sweep; *J (mask
// mode) receives the objective, *dJdhg dJ/dhgcoef; leaves the state at the
// final cycle.
int adjoint_run(const AdjointIO &io, double *J, double *dJdhg);

}  // namespace lg
