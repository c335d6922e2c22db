// phg_chs.cu -- Chebyshev solves of the mass-like operators in one persistent
// launch (Saad, Iterative Methods for Sparse Linear Systems, 2nd ed., Alg.
// 12.1, Jacobi-preconditioned, inside FP64 iterative refinement).
//
// A refinement cycle forms r = b - A x in FP64, runs Kc steps
//     d <- ca d + cb D^-1 (r - A e),  e <- e + d
// on r / ||r|| in the Krylov precision and adds ||r|| e to x.  A step is one
// gather of seven neighbours a row, so a single right-hand side is bound by
// the hand-over between steps and many by the FP64 (or gather) rate (against
// cheb_kernel, level 6 FP64: one 222 -> 90 us, the Jacobian's eight 554 -> 281):
//
//  * the iterate lives in stamped cells (phg_stamp.cuh): a row takes step k as
//    soon as its neighbours' step k - 1 is there, no barrier within a cycle;
//  * up to C right-hand sides of the operator advance together in one group of
//    blocks: the C values of a point sit side by side, so a gathered neighbour
//    is one contiguous piece and a row's entries are read once for all C;
//  * D^-1 A is stored by rows, the diagonal first: the row's own iterate comes
//    with the gather, and a block keeps its rows, d and r in shared memory.
//
// Two iterates' cells suffice: a row writes e_{k+1} over e_{k-1}, which is read
// only by rows that share an entry with it, when they compute e_k; it has seen
// e_k of all its neighbours by then, and these are the same rows because the
// pattern is symmetric (checked on the host; other operators keep cheb_kernel).
#include <cmath>
#include <cstring>
#include <mutex>

#include "phg_chs.cuh"
#include "phg_kernels.cuh"
#include "phg_stamp.cuh"

namespace phg {

namespace {

constexpr int RSC = 33;   // stride of the warps' partial sums

struct ChsParams {
    const int *col;            // exact A (FP64 residuals), slot-major
    const double *aval, *dinv;
    const int *c7;             // D^-1 A by rows of seven, the diagonal first
    const void *v7;
    int W, n, nv, ld, max_iter;
    double tol;
    const double *B;
    double *X;
    char *cells;               // per chunk of C right-hand sides: 2 n C cells
    void *dr;                  // per chunk: d and r, n C values each (when not in shared memory)
    double *R;                 // nv x n
    double *part;
    unsigned *bar;
    int *err;
    GmresStats *stats;
    int groups, G;
    int off_a, off_d, off_e;   // shared-memory byte offsets of the block's rows, of d and r, and (one block) of the
                               // two iterates; -1: global memory
    int K;
    double c0, lg, ils, two_tol;   // ils = 1 / ls, two_tol = 2 / tol
    double ca[CHEB_KMAX], cb[CHEB_KMAX];
    long long wait_limit;
};

template <typename VT, int C, bool ONE>
__global__ void __launch_bounds__(sizeof(VT) == 4 ? 1024 : 768, 1) chs_kernel(const __grid_constant__ ChsParams p) {
    using E = typename CellStore<VT, ONE>::E;
    using ST = CellStore<VT, ONE>;
    extern __shared__ __align__(16) char smem[];
    double *red = (double *)smem;                       // 2 C x RSC
    VT *cf = (VT *)(red + 2 * C * RSC);                 // ca, cb in the Krylov precision
    __shared__ double s_sum[2 * C], s_bn[C], s_bi[C], s_beta[C], s_prev[C], s_scale[C], s_rel[C];
    __shared__ int s_open[C], s_stat[C], s_iter[C], s_cyc[C], s_kc, s_dead;
    __shared__ long long s_since[32];

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, NT = blockDim.x, NW = NT >> 5;
    const int n = p.n, G = p.G, W = p.W, nv = p.nv;
    const size_t ld = (size_t)p.ld;
    const double tol = p.tol;
    const int grp = blockIdx.x / G, bi = blockIdx.x % G;
    if (grp >= p.groups) return;
    if (threadIdx.x == 0) {
        wait_limit_slot() = p.wait_limit;
        bar_epoch() = 0;
        s_dead = 0;
    }
    if (threadIdx.x < CHEB_KMAX) {
        cf[threadIdx.x] = (VT)p.ca[threadIdx.x];
        cf[CHEB_KMAX + threadIdx.x] = (VT)p.cb[threadIdx.x];
    }
    unsigned *bar = p.bar + 2 * grp;
    int *err = p.err;
    const Waits wt = {err, (unsigned long long *)bar, &s_dead, s_since, p.wait_limit};
    double *part2 = p.part + (size_t)(blockIdx.x - bi) * 2 * (MAXM + 2);
    int parity = 0;
    int r0, r1;
    own_rows(n, G, bi, r0, r1);
    const int cnt = r1 - r0, rpb = (n + G - 1) / G;
    const int NA = max(1, min(NW, (cnt + 31) / 32));    // warps with rows
    const int *__restrict__ col = p.col;
    const double *__restrict__ aval = p.aval;
    // the block's rows of D^-1 A
    const int *mc = p.c7 + (size_t)r0 * 7;
    const VT *mv = (const VT *)p.v7 + (size_t)r0 * 7;
    if (p.off_a >= 0) {
        VT *sv = (VT *)(smem + p.off_a);
        int *sc = (int *)(sv + (size_t)rpb * 7);
        for (int e = threadIdx.x; e < cnt * 7; e += NT) { sv[e] = mv[e]; sc[e] = mc[e]; }
        mc = sc;
        mv = sv;
    }
    const VT c0 = (VT)p.c0;
    unsigned ep = 0;           // stamp of the last iterate written
    // (FP64 scalars are one thread's business: the FP64 pipe takes 16 cycles per
    // warp instruction)
    int my_iters = 0, my_cycles = 0, my_status = 0, my_steps = 0, my_rsteps = 0, my_resid = 0, my_upd = 0;
    double my_rel = 0.0;

    for (int ch = grp; ch * C < nv; ch += p.groups) {
        const int v0 = ch * C, nc = min(C, nv - v0);
        E *e0 = ONE && p.off_e >= 0 ? (E *)(smem + p.off_e) : (E *)p.cells + (size_t)grp * 2 * n * C;
        E *e1 = e0 + (size_t)n * C;
        VT *d, *r;
        if (p.off_d >= 0) { d = (VT *)(smem + p.off_d); r = d + (size_t)rpb * C; }
        else { d = (VT *)p.dr + ((size_t)grp * 2 * n + r0) * C; r = d + (size_t)n * C; }
        if (!ONE && ep == 0)   // no stamp of an earlier launch survives (ordered by the first barrier below)
            for (int i = r0 * C + threadIdx.x; i < r1 * C; i += NT) { ST::put(e0 + i, (VT)0, 0u); ST::put(e1 + i, (VT)0, 0u); }
        if (threadIdx.x < C) {
            s_stat[threadIdx.x] = 0; s_iter[threadIdx.x] = 0; s_cyc[threadIdx.x] = 0;
            s_open[threadIdx.x] = threadIdx.x < nc; s_prev[threadIdx.x] = 0.0; s_rel[threadIdx.x] = 0.0;
        }
        __syncthreads();
        bool first = true;
        for (;;) {
            // R = b - A x (FP64, exact operator) and the norms, a thread per row
            double sr[8] = {0, 0, 0, 0, 0, 0, 0, 0}, sb[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll 1
            for (int i = r0 + threadIdx.x; i < r1; i += NT) {
                int c[8];
                double a[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    c[k] = k < W ? __ldg(&col[(size_t)k * n + i]) : i;
                    a[k] = k < W ? __ldg(&aval[(size_t)k * n + i]) : 0.0;
                }
#pragma unroll
                for (int v = 0; v < C; ++v) {
                    if (v >= nc || !s_open[v]) continue;
                    const double *x = p.X + (size_t)(v0 + v) * ld;
                    const double bv = p.B[(size_t)(v0 + v) * ld + i];
                    double t = 0.0, xv[7];
#pragma unroll
                    for (int k = 0; k < 7; ++k) xv[k] = ldcg(&x[c[k]]);
#pragma unroll
                    for (int k = 0; k < 7; ++k) t += a[k] * xv[k];
                    if (W > 7) t += a[7] * ldcg(&x[c[7]]);
                    const double q = bv - t;
                    p.R[(size_t)(v0 + v) * n + i] = q;
                    sr[v] += q * q;
                    if (first) sb[v] += bv * bv;
                }
            }
            if (warp < NA) {
                if constexpr (C == 1) {
                    sr[0] = warp_sum(sr[0]);
                    if (first) sb[0] = warp_sum(sb[0]);
                    if (lane == 0) { red[warp] = sr[0]; red[RSC + warp] = sb[0]; }
                } else {
                    const int k = lane >> 2;
                    const double q = fold8(sr, lane);
                    if ((lane & 3) == 0 && k < C) red[k * RSC + warp] = q;
                    if (first) {
                        const double t = fold8(sb, lane);
                        if ((lane & 3) == 0 && k < C) red[(C + k) * RSC + warp] = t;
                    }
                }
            }
            __syncthreads();
            double *part = part2 + (size_t)parity * G * (MAXM + 2);
            parity ^= 1;
            const int ns = first ? 2 * C : C;
#pragma unroll 1
            for (int l = warp; l < ns; l += NW) {
                double s = lane < NA ? red[l * RSC + lane] : 0.0;
                s = lanes_sum(s, NA);
                if (lane == 0) {
                    if (G == 1) s_sum[l] = s;
                    else part[(size_t)l * G + bi] = s;
                }
            }
            if (!group_sync(bar, G, err, nullptr)) return;
            if (G > 1) {
#pragma unroll 1
                for (int l = warp; l < ns; l += NW) {
                    double s = 0.0;
#pragma unroll 5
                    for (int q = lane; q < G; q += 32) s += ldcg(&part[(size_t)l * G + q]);
                    s = warp_sum(s);
                    if (lane == 0) s_sum[l] = s;
                }
                __syncthreads();
            }
            // the tests, one thread per right-hand side; steps of this cycle: K,
            // or fewer when the reduction still needed (tol / rel, with a
            // factor 2 margin) is smaller than the one K steps guarantee
            if (warp == 0) {
                int kc = 0;
                if (lane < nc && s_open[lane]) {
                    const double q = s_sum[lane], ri = q > 0.0 ? rsqrt(q) : 0.0, bt = q > 0.0 ? q * ri : q;
                    if (first) {
                        const double b2 = s_sum[C + lane], bi2 = b2 > 0.0 ? rsqrt(b2) : 0.0;
                        s_bn[lane] = b2 > 0.0 ? b2 * bi2 : b2;
                        s_bi[lane] = bi2;
                    }
                    const double bn = s_bn[lane], rl = bn > 0.0 ? bt * s_bi[lane] : (bn == 0.0 ? 0.0 : bn);
                    s_rel[lane] = rl;
                    int open = 1, stat = 0;
                    if (rl <= tol) open = 0;
                    else if (s_iter[lane] >= p.max_iter || (s_cyc[lane] > 0 && !(bt < 0.9999 * s_prev[lane]))) {
                        open = 0;
                        stat = 1;
                    }
                    s_stat[lane] = stat;
                    s_prev[lane] = bt;
                    s_beta[lane] = bt;
                    s_scale[lane] = ri;
                    s_open[lane] = open;
                    if (open) {
                        kc = p.K;
                        if (rl > tol && p.ils > 0.0) {
                            // whole steps: FP32 is enough for the count
                            const float need = ((float)p.lg + logf((float)(rl * p.two_tol))) * (float)p.ils;
                            if (need + 1.0f < (float)p.K) kc = max(2, (int)ceilf(need) + 1);
                        }
                    }
                }
                for (int o = 16; o > 0; o >>= 1) kc = max(kc, __shfl_xor_sync(0xffffffffu, kc, o));
                if (lane < nc && s_open[lane]) { s_cyc[lane] += 1; s_iter[lane] += kc; }
                if (lane == 0) s_kc = kc;
            }
            __syncthreads();
            ++my_resid;
            if (first) {   // zero right-hand sides: x = 0
#pragma unroll 1
                for (int v = 0; v < nc; ++v)
                    if (s_bn[v] == 0.0)
                        for (int i = r0 + threadIdx.x; i < r1; i += NT) p.X[(size_t)(v0 + v) * ld + i] = 0.0;
                first = false;
            }
            const int Kc = s_kc;
            if (Kc == 0) break;
            // e_1 = d_0 = c0 D^-1 r; r holds D^-1 r / ||r|| (zero for closed members)
#pragma unroll 1
            for (int i = threadIdx.x; i < cnt; i += NT) {
                const VT di = (VT)__ldg(&p.dinv[r0 + i]);
#pragma unroll
                for (int v = 0; v < C; ++v) {
                    VT q = 0;
                    if (v < nc && s_open[v]) q = (VT)(p.R[(size_t)(v0 + v) * n + r0 + i] * s_scale[v]) * di;
                    r[i * C + v] = q;
                    d[i * C + v] = c0 * q;
                    ST::put(e0 + (size_t)(r0 + i) * C + v, c0 * q, ep + 1);
                }
            }
            ++ep;
            __syncthreads();
            E *ec = e0, *en = e1;
#pragma unroll 1
            for (int k = 1; k < Kc; ++k) {
                const VT ca = cf[k], cb = cf[CHEB_KMAX + k];
#pragma unroll 1
                for (int t = warp * 32; t < cnt * C; t += NT) {
                    const int it = min(t + lane, cnt * C - 1), row = it / C, v = it % C;
                    const int *c_ = mc + row * 7;
                    const VT *a_ = mv + row * 7;
                    int c[7];
                    VT x[7];
#pragma unroll
                    for (int q = 0; q < 7; ++q) c[q] = c_[q] * C + v;
                    ST::get(x, ec, c, ep, wt);
                    VT s = r[it];
#pragma unroll
                    for (int q = 0; q < 7; ++q) s -= a_[q] * x[q];
                    const VT dd = ca * d[it] + cb * s;
                    if (t + lane < cnt * C) {
                        d[it] = dd;
                        ST::put(en + (size_t)r0 * C + it, x[0] + dd, ep + 1);
                    }
                }
                ++ep;
                if (ONE) __syncthreads();
                E *t = ec; ec = en; en = t;
            }
            for (int v = 0; v < nc; ++v) my_steps += s_open[v] ? Kc - 1 : 0;
            my_rsteps += Kc - 1;
            ++my_upd;
            if (__syncthreads_or(s_dead)) return;
            // x += ||r|| e
#pragma unroll 1
            for (int i = threadIdx.x; i < cnt; i += NT)
#pragma unroll
                for (int v = 0; v < C; ++v)
                    if (v < nc && s_open[v]) {
                        const VT e = ST::own(ec + (size_t)(r0 + i) * C + v);
                        p.X[(size_t)(v0 + v) * ld + r0 + i] += s_beta[v] * (double)e;
                    }
            if (!group_sync(bar, G, err, nullptr)) return;   // x complete
        }
        if (threadIdx.x == 0)
            for (int v = 0; v < nc; ++v) {
                my_iters = max(my_iters, s_iter[v]);
                my_cycles = max(my_cycles, s_cyc[v]);
                my_rel = max_nan(my_rel, s_rel[v]);
                my_status = max(my_status, s_stat[v]);
            }
        // the next chunk reuses the cells
        if ((ch + p.groups) * C < nv && !group_sync(bar, G, err, nullptr)) return;
    }
    if (threadIdx.x == 0) {   // algorithmic bytes: residuals, steps (rows once for the chunk), updates
        const double es = (double)sizeof(VT), c = min(C, nv);
        atomicAdd(&p.stats->bytes, (double)cnt * (my_resid * (W * 12.0 + 24.0 * c) + my_rsteps * 7.0 * (4.0 + es) +
                                                  my_steps * 7.0 * es + my_upd * c * (es + 16.0)));
    }
    if (threadIdx.x == 0 && bi == 0) {
        atomicAdd(&p.stats->steps_total, my_steps);
        atomicMax(&p.stats->iters, my_iters);
        atomicMax(&p.stats->cycles, my_cycles);
        atomicMax(&p.stats->status, my_status);
        atomicMax((unsigned long long *)&p.stats->relres, (unsigned long long)__double_as_longlong(my_rel));
    }
}

using Kernel = void (*)(const ChsParams);

template <typename VT, bool ONE> Kernel chs_fn_c(int C) {
    return C == 1 ? chs_kernel<VT, 1, ONE> : C == 2 ? chs_kernel<VT, 2, ONE>
         : C == 4 ? chs_kernel<VT, 4, ONE> : chs_kernel<VT, 8, ONE>;
}
Kernel chs_fn(Precision prec, int C, bool one) {
    if (prec == PREC_MIXED) return one ? chs_fn_c<float, true>(C) : chs_fn_c<float, false>(C);
    return one ? chs_fn_c<double, true>(C) : chs_fn_c<double, false>(C);
}

// bytes of dynamic shared memory a block may take (set once per kernel)
cudaError_t chs_smem_limit(Precision prec, int C, bool one, int *limit) {
    static std::once_flag once[2][8];
    static cudaError_t err[2][8];
    static int lim[2][8];
    const int a = prec == PREC_MIXED ? 1 : 0, b = (C == 1 ? 0 : C == 2 ? 1 : C == 4 ? 2 : 3) + (one ? 4 : 0);
    std::call_once(once[a][b], [&] {
        int dev = 0, optin = 0;
        cudaFuncAttributes fa;
        const void *fn = (const void *)chs_fn(prec, C, one);
        if ((err[a][b] = cudaGetDevice(&dev)) != cudaSuccess) return;
        if ((err[a][b] = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess)
            return;
        if ((err[a][b] = cudaFuncGetAttributes(&fa, fn)) != cudaSuccess) return;
        lim[a][b] = optin - (int)fa.sharedSizeBytes;
        err[a][b] = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, lim[a][b]);
    });
    *limit = lim[a][b];
    return err[a][b];
}

// Small systems run in one block each (no hand-over between blocks): a step
// costs their own work there, about 1.6 cycles a row in FP32 (shared-memory
// loads) and 5.5 in FP64 (multiply-adds), against 1,400 to 1,800 cycles for a
// hand-over.  Level 3 (641 rows), mixed: one Laplacian apply 94 -> 80 us, and
// level 4 (2,561) the other way, 92 against 154 us.
bool small_system(int n, Precision prec) { return n <= (prec == PREC_MIXED ? 1000 : 300); }

// right-hand sides per chunk: side by side in one group of blocks, up to
// eight; small systems only as many as leave every chunk a block of its own
int chunk_of(int n, int nv, Precision prec, int sms) {
    int C = 1;
    if (small_system(n, prec))
        while (C < 8 && (nv + C - 1) / C > sms) C *= 2;
    else
        while (C < 8 && C < nv) C *= 2;
    return C;
}

}  // namespace

size_t chs_work_bytes(const DevSolveOp &op, int nv, Precision prec, int sms) {
    const int C = chunk_of(op.A.n, nv, prec, sms), chunks = std::min((nv + C - 1) / C, sms);
    const size_t per = 2 * (size_t)op.A.n * C * chunks;
    auto al = [](size_t b) { return (b + 255) & ~size_t(255); };
    return al(per * (prec == PREC_MIXED ? 8 : 16)) + al(per * (prec == PREC_MIXED ? 4 : 8));
}

cudaError_t chs_prepare() {
    int lim;
    cudaError_t e = cudaSuccess;
    for (Precision prec : {PREC_FP64, PREC_MIXED})
        for (int C : {1, 2, 4, 8})
            for (bool one : {false, true})
                if (e == cudaSuccess) e = chs_smem_limit(prec, C, one, &lim);
    return e;
}

cudaError_t chs_solve(const DevSolveOp &op, const ChsArgs &q, cudaStream_t s) {
    const int n = op.A.n, C = chunk_of(n, q.nv, q.prec, q.sms), chunks = (q.nv + C - 1) / C;
    const size_t es = q.prec == PREC_MIXED ? 4 : 8;
    const int sms = (q.max_sms > 0 && q.max_sms < q.sms) ? q.max_sms : q.sms;
    // one block per SM, shared out over the chunks; two smaller ones where the
    // caller leaves this launch a part of the SMs (see mgs_solve)
    const bool half = sms < q.sms;
    const int slots = half ? 2 * sms : sms, groups = std::min(chunks, std::min(slots, q.sms));
    int G = slots / groups;
    if (q.rpb > 0) G = std::min(G, (n + q.rpb - 1) / q.rpb);
    if (small_system(n, q.prec)) G = 1;
    G = std::max(G, 1);
    const bool one = G == 1;
    int limit = 0;
    cudaError_t e = chs_smem_limit(q.prec, C, one, &limit);
    if (e != cudaSuccess) return e;
    if (half) limit = std::min(limit, 104 * 1024);
    ChsParams p;
    memset(&p, 0, sizeof p);
    const size_t rpb = (size_t)((n + G - 1) / G);
    size_t used = (sizeof(double) * 2 * C * RSC + es * 2 * CHEB_KMAX + 15) & ~size_t(15);
    auto take = [&](size_t bytes) -> int {
        bytes = (bytes + 15) & ~size_t(15);
        if (used + bytes > (size_t)limit) return -1;
        const int o = (int)used;
        used += bytes;
        return o;
    };
    p.off_d = take(2 * es * rpb * C);
    p.off_e = one ? take(2 * es * rpb * C) : -1;
    p.off_a = take(rpb * 7 * (es + 4));
    p.col = op.A.col; p.aval = op.A.val; p.dinv = op.dinv; p.c7 = op.c7; p.v7 = op.v7;
    p.W = op.A.W; p.n = n; p.nv = q.nv; p.ld = q.ld; p.max_iter = q.max_iter; p.tol = q.tol;
    p.B = q.B; p.X = q.X; p.R = q.R;
    p.cells = (char *)q.work;
    const size_t per = 2 * (size_t)n * C * std::min(chunks, q.sms);
    p.dr = (char *)q.work + ((per * (q.prec == PREC_MIXED ? 8 : 16) + 255) & ~size_t(255));
    p.part = q.part; p.bar = q.bar; p.err = &q.stats->status; p.stats = q.stats;
    p.groups = groups; p.G = G;
    p.K = q.plan->K; p.c0 = q.plan->c0; p.lg = q.plan->lg; p.ils = q.plan->ls > 0.0 ? 1.0 / q.plan->ls : 0.0; p.two_tol = 2.0 / q.tol;
    memcpy(p.ca, q.plan->ca, sizeof p.ca);
    memcpy(p.cb, q.plan->cb, sizeof p.cb);
    p.wait_limit = q.wait_limit;
    // threads for a row and right-hand side each, as far as there are
    const int most = half ? 384 : q.prec == PREC_MIXED ? 1024 : 768;
    const int threads = (int)std::min<size_t>(most, std::max<size_t>(256, (rpb * C + 31) / 32 * 32));
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute coop[1];
    coop[0].id = cudaLaunchAttributeCooperative;
    coop[0].val.cooperative = 1;
    cfg.gridDim = dim3(groups * G);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = used;
    cfg.stream = s;
    cfg.attrs = coop;
    cfg.numAttrs = 1;
    void *args[] = {&p};
    if ((e = cudaLaunchKernelExC(&cfg, (const void *)chs_fn(q.prec, C, one), args)) != cudaSuccess) return e;
    ++g_kernel_launches;
    return cudaGetLastError();
}

}  // namespace phg
