// phg_chs.cuh -- the launcher of the persistent Chebyshev solves.
#pragma once
#include "phg_device.cuh"

namespace phg {

constexpr int CHEB_KMAX = 64;    // most Chebyshev steps per refinement cycle

// The recurrence d_k = ca[k] d_{k-1} + cb[k] D^-1 r_k, d_0 = c0 D^-1 r_0 on the
// operator's spectrum interval; K steps reduce the residual by eps, and a
// reduction e takes ceil((lg - log e) / ls) + 1 steps.
struct ChebPlan {
    int K;
    double c0, lg, ls;
    double ca[CHEB_KMAX], cb[CHEB_KMAX];
};
void cheb_plan(const DevSolveOp &op, double eps, ChebPlan &p);

struct ChsArgs {
    const double *B;
    double *X;
    int nv, ld, max_iter;
    double tol;
    Precision prec;
    const ChebPlan *plan;
    int rpb;               // rows per block at least (0 = no limit)
    int sms, max_sms;
    long long wait_limit;
    void *work;            // chs_work_bytes
    double *R;             // nv x n
    double *part;          // partial sums of the blocks
    unsigned *bar;         // zeroed before the launch
    GmresStats *stats;     // zeroed before the launch; its status is the launch's error flag
};

size_t chs_work_bytes(const DevSolveOp &op, int nv, Precision prec, int sms);
// load every instantiation (operator creation calls it): the first launch of a
// kernel that is loaded then waits for the device, and so for other streams' work
cudaError_t chs_prepare();
cudaError_t chs_solve(const DevSolveOp &op, const ChsArgs &a, cudaStream_t s);

}  // namespace phg
