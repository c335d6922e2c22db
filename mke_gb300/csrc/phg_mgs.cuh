// phg_mgs.cuh -- the launcher of the Laplacian's persistent multigrid solves.
#pragma once
#include "phg_device.cuh"

namespace phg {

struct MgsArgs {
    const double *B;
    double *X;
    int nv, ld, m, max_iter;
    double tol, inner_rtol;
    Precision prec;
    int rpb;               // rows per block at least (0 = no limit)
    int sms, max_sms;
    long long wait_limit;
    void *V, *Z, *Wv;      // nv x (m + 1) x n, nv x m x n, nv x n in the Krylov precision
    double *R;             // nv x n
    void *scratch;         // min(nv, GROUPS_CAP) x mgs_scratch_bytes
    double *part;          // partial sums of the blocks
    unsigned *bar;         // zeroed before the launch
    GmresStats *stats;     // zeroed before the launch; its status is the launch's error flag
};

bool mgs_applicable(const DevSolveOp &op);
size_t mgs_scratch_bytes(const DevSolveOp &op, Precision prec);   // per right-hand side in flight
// load every instantiation (operator creation calls it): the first launch of a
// kernel that is loaded then waits for the device, and so for other streams' work
cudaError_t mgs_prepare();
cudaError_t mgs_solve(const DevSolveOp &op, const MgsArgs &a, cudaStream_t s);

}  // namespace phg
