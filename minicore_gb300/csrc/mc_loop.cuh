// State of the device-side Lloyd loop and the two decisions that kernels of the loop take at their
// end: the stop rule where the objective's sum is finished, the search for empty clusters where the
// bucket sizes are (as launches of their own the two cost 1.6 and 2.8 us per update, all latency).
#pragma once
#include "mc_internal.cuh"

namespace mc {

enum : int { LOOP_RUN = 0, LOOP_DONE = 1, LOOP_REVERT = 2, LOOP_EMPTY = 3, LOOP_NAN = 4, LOOP_TIMEOUT = 5 };

struct LoopState {
    float cost;                  // objective of the committed centers C
    int reason;                  // LOOP_*
    unsigned long long iternum;  // committed updates
    unsigned long long maxiter;
    double eps;
    int commit;                  // the last decision copies Cw to C
    int pad;
};

struct LoopCtl {
    LoopState *ls = nullptr;  // null: the kernel decides nothing
    int *nan_flag = nullptr;  // zero again after a decision
    const int *tc_err = nullptr;
    cudaGraphConditionalHandle h{};
    int graph = 0;  // the kernel runs inside the loop graph and also sets its while-condition h
};

#ifdef __CUDACC__
// a cluster is empty: the host restarts it (one thread)
__device__ inline void loop_empty(const LoopCtl &c) {
    if (c.ls->reason != LOOP_RUN) return;
    c.ls->reason = LOOP_EMPTY;
    if (c.graph) cudaGraphSetConditional(c.h, 0);
}

// the stop rule of the host loop (perform_hard_clustering, clustering/solve.h:98-175) (one thread)
__device__ inline void loop_decide(const LoopCtl &c, double cost_sum) {
    LoopState *ls = c.ls;
    ls->commit = 0;
    if (*c.nan_flag) {
        *c.nan_flag = 0;
        ls->reason = LOOP_NAN;
        if (c.graph) cudaGraphSetConditional(c.h, 0);
        return;
    }
    if (c.tc_err && *c.tc_err) {
        ls->reason = LOOP_TIMEOUT;
        if (c.graph) cudaGraphSetConditional(c.h, 0);
        return;
    }
    const float newcost = float(cost_sum);
    if (newcost > ls->cost) {
        ls->reason = LOOP_REVERT;
        if (c.graph) cudaGraphSetConditional(c.h, 0);
        return;
    }
    ls->commit = 1;
    ls->iternum += 1;
    const float oldcost = ls->cost;
    ls->cost = newcost;
    const double mx = double(newcost) < double(oldcost) ? double(oldcost) : double(newcost);
    if (double(oldcost - newcost) < ls->eps * mx || ls->iternum > ls->maxiter) {
        ls->reason = LOOP_DONE;
        if (c.graph) cudaGraphSetConditional(c.h, 0);
    } else {
        if (c.graph) cudaGraphSetConditional(c.h, 1);
    }
}
#endif

}  // namespace mc
