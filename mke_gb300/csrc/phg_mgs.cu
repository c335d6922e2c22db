// phg_mgs.cu -- the Laplacian's multigrid solves: restarted FGMRES with a
// V-cycle as right preconditioner, in one persistent launch per call.
//
// A group of blocks owns one right-hand side at a time and splits every
// level's rows; the algorithm, the stopping tests and the FP64 refinement loop
// are gmres_kernel's (phg_gmres.cu).  What bounds a single solve is latency --
// a level-6 vector is 160 KB -- so the kernel is built to have few dependent
// phases per Arnoldi step and cheap hand-overs between them (one solve, against
// gmres_kernel: level 3 FP64 910 -> 255 us, level 7 mixed 3.73 -> 0.85 ms):
//
//  * the V-cycle runs as composed operators (phg_mgplan.cpp): one gather per
//    level down (b' = Q b) and one up (x = T b + U x'), the small levels as one
//    dense product, and A z formed with z from the same gather: 6 phases per
//    V-cycle and apply at level 6, where the level-by-level cycle and the apply
//    have twelve group barriers;
//  * gathered vectors live in stamped cells (phg_stamp.cuh): a row waits for
//    its neighbours' values, not for a barrier over all blocks; the sums of
//    the dot products are published and collected the same way;
//  * each block keeps its own rows of every operator, and of the Krylov
//    vectors as far as they fit, in shared memory: after a barrier or an
//    acquire the L1 is empty, and a row's index load would add a round trip to
//    L2 to every phase;
//  * the Krylov vector is normalised after the V-cycle, which is linear: the
//    norm's sum and the rotations run on a warp of their own (the helper) while
//    the other warps are already in the next V-cycle.  The stopping test comes
//    out of it too, so the last step's V-cycle is begun once in vain.
//
// The baroclinic block system (BLK; unknown 4i + q of vertex i, w1 w2 u1 u2) runs
// through the same kernel: its preconditioner z_w = D^-1 v_w, z_u = -V(v_u - M z_w)
// is one V-cycle of two vectors at once (C = 2, side by side), and its apply
// needs no gather of z: the w rows' mass-like part comes with M z_w from the
// gather of v, the u rows are M z_w - L z_u = M z_w + L V(t), which the
// finest level's last gather gives as for one Laplacian, and u2's part of the
// w2 rows is composed with it in the same way.
//
// Why no cell is overwritten too early: a block writes the cells of Arnoldi
// step j + 1 only after it has collected the dot products of step j from every
// block, and a block publishes its part of those after its own gathers of step
// j.  The Krylov vector's cells are written after the collection of step j and
// read before the publication of step j + 1.
#include <cmath>
#include <cstring>
#include <mutex>

#include "phg_kernels.cuh"
#include "phg_mgs.cuh"
#include "phg_stamp.cuh"

namespace phg {

namespace {

constexpr int RS = 33;           // stride of the warps' partial sums (up to 32 warps)
constexpr int NB = 5;            // published sums a lane collects at a time
constexpr int N_TAB = 3 * MG_MAXLEV + 2;
enum { TAB_Q = 0, TAB_T = MG_MAXLEV, TAB_U = 2 * MG_MAXLEV, TAB_F = 3 * MG_MAXLEV, TAB_C = 3 * MG_MAXLEV + 1 };

// a sparse operator: entries and values of all rows in global memory, and the
// shared-memory offsets of a block's own rows (off < 0: not copied)
struct Table {
    const void *c, *v, *v2, *v3;
    int rows, off, off2, off3, offc;
};
// a block's rows of `words` 32-bit words each, copied to shared memory at dst
struct Copy {
    const void *src;
    int rows, words, dst;
};

struct MgsParams {
    int x_n[MG_MAXLEV];        // rows of the levels
    const int *col;            // finest level: exact A (FP64 residuals)
    const double *aval;
    int W, n, nv, ld, m, max_iter;   // n: rows of the finest level (vertices of a block system)
    const double *dinv;        // block system: 1 / diagonal
    double tol, inner_rtol;
    const double *B;
    double *X;
    void *V, *Z, *Wv;
    double *R;
    void *scratch;             // groups x group_bytes: the cells
    size_t group_bytes;
    double *part;
    char *cpart;               // stamped partial sums, (MAXM + 2) x blocks
    unsigned *bar;
    int *err;
    GmresStats *stats;
    int groups, G;
    int top, bot;              // the dense product gives x on level top from b on level bot
    double step_row_bytes, resid_row_bytes;
    long long wait_limit;
    size_t boff[MG_MAXLEV], xoff[MG_MAXLEV];   // cell offsets of b_l and x_l (l >= 1)
    Table tab[N_TAB];
    Copy copy[4 * N_TAB];
    int ncopy;
    const void *dense, *dense2;
    int off_d, off_d2;         // the dense rows in shared memory (-1: in global memory)
    int off_w, off_t, off_v;   // own rows of A z (-1: in Wv), of T b (-1: not kept), of the Krylov vectors
    int mv, mvp;               // Krylov vectors kept in shared memory, and the rows there are for them
    int off_b;                 // the dense product's input
};

// this block's rows of one sparse operator: row i at c, v + (i - base) * stride
template <typename VT> struct Rows {
    const int *c;
    const VT *v, *v2, *v3;
    int base;
};

// sum over N entries of a row, KS apart: v[k] x[C c[k]] (C vectors side by side)
template <typename VT, bool ONE, int N, int KS, int C>
__device__ __forceinline__ VT row_sum(const int *col, const VT *v, const typename CellStore<VT, ONE>::E *p, unsigned stamp,
                                      const Waits &w) {
    int c[N];
    VT x[N];
#pragma unroll
    for (int q = 0; q < N; ++q) c[q] = C * col[KS * q];
    CellStore<VT, ONE>::get(x, p, c, stamp, w);
    VT s = 0, t = 0;   // two chains: a dependent FP64 multiply-add takes 81 cycles
#pragma unroll
    for (int q = 0; q < N; ++q) {
        if (sizeof(VT) == 8 && (q & 1)) t += v[KS * q] * x[q];
        else s += v[KS * q] * x[q];
    }
    return sizeof(VT) == 8 ? s + t : s;
}

// a dense row (16-byte aligned, length a multiple of four) times b, in every lane
template <typename VT>
__device__ __forceinline__ VT dense_row(const VT *row, const VT *b, int len, int lane) {
    VT s = 0, s1 = 0, s2 = 0, s3 = 0;
    if constexpr (sizeof(VT) == 4) {
#pragma unroll 3
        for (int k = lane; k < len / 4; k += 32) {
            const float4 a = ((const float4 *)row)[k], x = ((const float4 *)b)[k];
            s += a.x * x.x; s1 += a.y * x.y; s += a.z * x.z; s1 += a.w * x.w;
        }
    } else {
#pragma unroll 2
        for (int k = lane; k < len / 2; k += 64) {
            const double2 a = ((const double2 *)row)[k], x = ((const double2 *)b)[k];
            s += a.x * x.x; s1 += a.y * x.y;
            if (k + 32 < len / 2) {
                const double2 c = ((const double2 *)row)[k + 32], z = ((const double2 *)b)[k + 32];
                s2 += c.x * z.x; s3 += c.y * z.y;
            }
        }
    }
    return warp_sum((s + s1) + (s2 + s3));
}

// Sums over the group's blocks, the same bits in every block.  Each block
// publishes its part of a value; one block per value (its root) collects them
// and publishes the sum, which every block reads: two hand-overs, but each
// cell is waited for by few.  Letting every block collect all parts takes one
// hand-over and 152 x 152 waiting loads per value, and measured four times as
// long (10,000 cycles a step against 3,900).
// The root's part, by one warp: the sum over the G published parts.
template <typename VT>
__device__ __noinline__ VT root_sum(const Cell<VT> *part, int G, unsigned stamp, const Waits &w) {
    const int lane = threadIdx.x & 31;
    VT s = 0;
#pragma unroll 1
    for (int b0 = 0; b0 < G; b0 += 32 * NB) {
        int c[NB];
        VT t[NB];
#pragma unroll
        for (int q = 0; q < NB; ++q) c[q] = min(b0 + lane + 32 * q, G - 1);
        wait_cells<VT, NB>(t, part, c, stamp, w);
#pragma unroll
        for (int q = 0; q < NB; ++q)
            if (b0 + lane + 32 * q < G) s += t[q];
    }
    return warp_sum(s);
}

// BLK: the block system of four unknowns per vertex (C = 2 vectors per V-cycle)
template <typename VT, bool ONE, bool BLK>
__global__ void __launch_bounds__(sizeof(VT) == 4 ? 800 : 544, 1) mgs_kernel(const __grid_constant__ MgsParams p) {
    using ST = CellStore<VT, ONE>;
    using E = typename ST::E;
    constexpr int C = BLK ? 2 : 1, NK = BLK ? 4 : 1;   // vectors per V-cycle, Krylov entries per finest row
    extern __shared__ __align__(16) char smem[];
    double *H = (double *)smem;              // (m + 1) x m, the R factor
    double *cs = H + (MAXM + 1) * MAXM, *sn = cs + MAXM, *g = sn + MAXM, *y = g + MAXM + 1;
    double *hcol = y + MAXM;                 // the current column
    double *red = hcol + MAXM + 2;           // (MAXM + 2) x RS partial sums of the warps
    VT *redv = (VT *)red;                    // the same in the Krylov precision
    VT *hv = (VT *)(red + (MAXM + 2) * RS);  // the column in the Krylov precision
    __shared__ Rows<VT> tab[N_TAB];
    __shared__ double scal[5], s_a, s_target;
    __shared__ VT s_inv;
    __shared__ int s_stop, s_dead, s_go, s_zero;
    __shared__ long long s_since[32];

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int NW = (blockDim.x >> 5) - 1;    // worker warps; the last warp is the helper
    const bool helper = warp == NW;
    const int m = p.m, n = p.n, W = p.W, G = p.G, max_iter = p.max_iter, top = p.top, bot = p.bot;
    const size_t ld = (size_t)p.ld;
    const double tol = p.tol;
    const int grp = blockIdx.x / G, bi = blockIdx.x % G;
    if (grp >= p.groups) return;
    unsigned *bar = p.bar + 2 * grp;
    int *err = p.err;
    const Waits wt = {err, (unsigned long long *)bar, &s_dead, s_since, p.wait_limit};
    if (threadIdx.x == 0) {
        wait_limit_slot() = p.wait_limit;
        bar_epoch() = 0;
        s_dead = 0;
    }
    double *part2 = p.part + (size_t)(blockIdx.x - bi) * 2 * (MAXM + 2);
    // published parts [value][block of the group] and sums [value]; the values
    // are the column's dot products and, last, the norm
    E *cpart = (E *)p.cpart + (size_t)(blockIdx.x - bi + grp) * (MAXM + 2);
    E *csum = cpart + (size_t)(MAXM + 2) * G;
    const int root_norm = G / 2;
    int parity = 0;
    int r0, r1;
    own_rows(n, G, bi, r0, r1);
    const int *__restrict__ col = p.col;
    const double *__restrict__ aval = p.aval;
    E *cw = (E *)((char *)p.scratch + (size_t)grp * p.group_bytes);   // Krylov vector (not normalised)
    E *ct = cw + (size_t)NK * n;                                       // T b of the finest level
    E *c0 = BLK ? ct + (size_t)C * n : cw;                             // b of the finest level
    E *cells = cw;
    VT *Vp = (VT *)p.V, *Zp = (VT *)p.Z;
    const double es = (double)sizeof(VT);
    const double inner_rtol = sizeof(VT) == 4 ? p.inner_rtol : 0.0;

    // ---- this block's rows of the operators: copied into shared memory where
    // the plan says so, and where each table's rows are
#pragma unroll 1
    for (int k = 0; k < p.ncopy; ++k) {
        const Copy &c = p.copy[k];
        int i0, i1;
        own_rows(c.rows, G, bi, i0, i1);
        const int *src = (const int *)c.src + (size_t)i0 * c.words;
        const unsigned dst = (unsigned)__cvta_generic_to_shared(smem + c.dst);
        const int words = (i1 - i0) * c.words;
#pragma unroll 4
        for (int e = threadIdx.x; e < words; e += blockDim.x)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + 4 * e), "l"(src + e) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (threadIdx.x < N_TAB) {
        const Table &t = p.tab[threadIdx.x];
        int i0 = 0, i1;
        Rows<VT> A = {(const int *)t.c, (const VT *)t.v, (const VT *)t.v2, (const VT *)t.v3, 0};
        if (t.off >= 0) {
            own_rows(t.rows, G, bi, i0, i1);
            A.v = (const VT *)(smem + t.off);
            A.v2 = (const VT *)(smem + t.off2);
            A.v3 = (const VT *)(smem + t.off3);
            A.c = (const int *)(smem + t.offc);
            A.base = i0;
        }
        tab[threadIdx.x] = A;
    }
    // the dense rows (level top), and A times them when top is the finest
    const int nb = p.x_n[bot];
    int d0, d1;
    own_rows(p.x_n[top], G, bi, d0, d1);
    const int nbs = mgx_stride(nb);   // row stride, padded with zeros
    const VT *dn = p.off_d >= 0 ? (const VT *)(smem + p.off_d) : (const VT *)p.dense + (size_t)d0 * nbs;
    const VT *dn2 = p.off_d >= 0 ? (const VT *)(smem + p.off_d2) : (const VT *)p.dense2 + (size_t)d0 * nbs;
    VT *bsm = (VT *)(smem + p.off_b);
    VT *vsm = (VT *)(smem + p.off_v);
    const int rpb = NK * ((n + G - 1) / G), nk = NK * n;    // Krylov entries of a block, and in all
    const int k0 = NK * r0, kn = NK * (r1 - r0);            // this block's
    const int NA = max(1, min(NW, (kn + 31) / 32));         // worker warps with Krylov entries
    if (!ONE) {   // no stamp of an earlier launch survives (ordered by the first barrier below)
#pragma unroll 1
        for (int i = k0 + threadIdx.x; i < k0 + kn; i += blockDim.x) ST::put(cw + i, (VT)0, 0u);
#pragma unroll 1
        for (int i = C * r0 + threadIdx.x; i < C * r1; i += blockDim.x) {
            ST::put(ct + i, (VT)0, 0u);
            if (BLK) ST::put(c0 + i, (VT)0, 0u);
        }
#pragma unroll 1
        for (int l = 1; l <= bot; ++l) {
            int i0, i1;
            own_rows(p.x_n[l], G, bi, i0, i1);
#pragma unroll 1
            for (int i = C * i0 + threadIdx.x; i < C * i1; i += blockDim.x) {
                ST::put(cells + p.boff[l] + i, (VT)0, 0u);
                ST::put(cells + p.xoff[l] + i, (VT)0, 0u);
            }
        }
#pragma unroll 1
        for (int l = threadIdx.x; l < MAXM + 2; l += blockDim.x) {
            ST::put(cpart + (size_t)l * G + bi, (VT)0, 0u);
            if (bi == 0) ST::put(csum + l, (VT)0, 0u);
        }
    }
    for (int k = nb + threadIdx.x; k < nbs; k += blockDim.x)
        for (int q = 0; q < C; ++q) bsm[q * nbs + k] = (VT)0;
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();

    // Scalars in FP64 are one thread's business: the FP64 pipe takes 16 cycles
    // per warp instruction, so a sum kept or a test made by all 25 warps costs as
    // much as a hand-over.  Thread 0 decides a cycle's start (s_go); the byte
    // count is formed from counters at the end.
    int my_iters = 0, my_cycles = 0, my_status = 0, my_steps = 0, my_resid = 0, my_cols = 0;
    double my_rel = 0.0;
    unsigned ep = 0;           // stamp of the current V-cycle

#pragma unroll 1
    for (int v = grp; v < p.nv; v += p.groups) {
        const double *__restrict__ b = p.B + (size_t)v * ld;
        double *x = p.X + (size_t)v * ld;
        VT *V = Vp + (size_t)v * (m + 1) * nk, *Z = Zp + (size_t)v * m * nk;
        VT *wl = p.off_w >= 0 ? (VT *)(smem + p.off_w) : (VT *)p.Wv + (size_t)v * nk + k0;   // own rows of A z
        VT *tl = p.off_t >= 0 ? (VT *)(smem + p.off_t) : nullptr;   // own rows of T b (null: read from ct)
        double *R = p.R + (size_t)v * nk;
        // own rows of Krylov vector l
        auto vrow = [&](int l) -> VT * { return l < p.mv ? vsm + (size_t)l * rpb : V + (size_t)l * nk + k0; };
        int iters = 0, cycles = 0;
        double beta_prev = 0.0;   // thread 0's
#pragma unroll 1
        for (;;) {
            // r = b - A x (FP64, exact operator) and its norm; with ||b|| the first time
            {
                double sb = 0.0, sr = 0.0;
                if (!helper)
#pragma unroll 1
                    for (int i = k0 + threadIdx.x; i < k0 + kn; i += NW * 32) {
                        double t = 0.0;
#pragma unroll 1
                        for (int w0 = 0; w0 < W; w0 += 8) {
                            int c[8];
                            double a[8], xv[8];
#pragma unroll
                            for (int k = 0; k < 8; ++k)
                                if (w0 + k < W) {
                                    c[k] = __ldg(&col[(size_t)(w0 + k) * nk + i]);
                                    a[k] = __ldg(&aval[(size_t)(w0 + k) * nk + i]);
                                }
#pragma unroll
                            for (int k = 0; k < 8; ++k)
                                if (w0 + k < W) xv[k] = ldcg(&x[c[k]]);
#pragma unroll
                            for (int k = 0; k < 8; ++k)
                                if (w0 + k < W) t += a[k] * xv[k];
                        }
                        const double bv = b[i], q = bv - t;
                        R[i] = q;
                        sr += q * q;
                        if (cycles == 0) sb += bv * bv;
                    }
                if (warp < NA) {
                    sr = warp_sum(sr);
                    if (cycles == 0) sb = warp_sum(sb);
                    if (lane == 0) { red[warp] = sr; red[RS + warp] = sb; }
                }
                __syncthreads();
                double *part = part2 + (size_t)parity * G * (MAXM + 2);
                parity ^= 1;
                if (warp < 2) {
                    double s = lane < NA ? red[warp * RS + lane] : 0.0;
                    s = lanes_sum(s, NA);
                    if (lane == 0) part[(size_t)warp * G + bi] = s;
                }
                if (!group_sync(bar, G, err, nullptr)) return;
                if (warp < 2) {
                    double s = 0.0;
#pragma unroll 5
                    for (int q = lane; q < G; q += 32) s += ldcg(&part[(size_t)warp * G + q]);
                    s = warp_sum(s);
                    if (lane == 0) hcol[warp] = s;
                }
                __syncthreads();
            }
            if (threadIdx.x < 2) {   // ||r|| and, the first time, ||b|| with their reciprocals, side by side
                const double q = hcol[threadIdx.x], ri = q > 0.0 ? rsqrt(q) : 0.0;
                const double nrm = q > 0.0 ? q * ri : q;   // NaN stays NaN
                if (threadIdx.x == 0) { scal[1] = nrm; scal[3] = ri; }
                else if (cycles == 0) { scal[0] = nrm; scal[4] = ri; }
                __syncwarp(3u);
                if (threadIdx.x == 0) {
                    const double bn = scal[0];
                    const double rel = bn > 0.0 ? nrm * scal[4] : (bn == 0.0 ? 0.0 : bn);
                    s_target = fmax(tol * bn, inner_rtol * nrm);
                    g[0] = nrm;
                    int go = 1, status = 0;
                    if (rel <= tol) go = 0;   // also a zero right-hand side
                    else if (iters >= max_iter || (cycles > 0 && !(nrm < 0.9999 * beta_prev))) { go = 0; status = 1; }
                    beta_prev = nrm;
                    s_go = go;
                    s_zero = bn == 0.0;
                    if (!go) {
                        my_rel = max_nan(my_rel, rel);
                        my_status = max(my_status, status);
                    }
                }
            } else if (threadIdx.x >= 32 && threadIdx.x < 32 + m) {
                g[threadIdx.x - 31] = 0.0;
            }
            __syncthreads();
            ++my_resid;
            if (s_zero)
#pragma unroll 1
                for (int i = k0 + threadIdx.x; i < k0 + kn; i += blockDim.x) x[i] = 0.0;
            if (!s_go) break;
            ++cycles;
            if (!helper) {
                const double ib = scal[3];
                VT *v0 = vrow(0);
#pragma unroll 1
                for (int i = threadIdx.x; i < kn; i += NW * 32) {
                    const VT q = (VT)(R[k0 + i] * ib);
                    v0[i] = q;
                    ST::put(cw + k0 + i, q, ep + 1);
                }
            }
            if (ONE) __syncthreads();

            int jl = 0;
#pragma unroll 1
            for (int j = 0;; ++j) {
                ++ep;
                if (helper) {
                    // norm of the last step's vector, its rotation and the stopping test
                    if (j > 0) {
                        if (!ONE) asm volatile("bar.sync 1, %0;" ::"r"((int)blockDim.x) : "memory");
                        double s = lane < NA ? (double)redv[lane] : 0.0;
                        s = lanes_sum(s, NA);
                        VT q = (VT)s;
                        if constexpr (!ONE) {
                            E *np = cpart + (size_t)(MAXM + 1) * G, *ns = csum + MAXM + 1;
                            if (lane == 0) ST::put(np + bi, q, ep);
                            if (bi == root_norm) {
                                q = root_sum<VT>(np, G, ep, wt);
                                if (lane == 0) ST::put(ns, q, ep);
                            } else {
                                const int c[1] = {0};
                                VT t[1];
                                ST::get(t, ns, c, ep, wt);
                                q = t[0];
                            }
                        }
                        if (lane == 0) {
                            const double hn2 = (double)q, a = s_a;
                            const double ri = hn2 > 0.0 ? rsqrt(hn2) : 0.0;
                            const double hn = hn2 > 0.0 ? hn2 * ri : hn2;   // NaN stays NaN
                            const double r2 = a * a + hn2;
                            const double ir = r2 > 0.0 ? rsqrt(r2) : 0.0, r = r2 > 0.0 ? r2 * ir : r2;
                            const int k = j - 1;
                            cs[k] = r > 0.0 ? a * ir : 1.0;
                            sn[k] = r > 0.0 ? hn * ir : 0.0;
                            H[k * MAXM + k] = r;
                            g[k + 1] = -sn[k] * g[k];
                            g[k] = cs[k] * g[k];
                            s_inv = (VT)ri;
                            s_stop = fabs(g[k + 1]) <= s_target || hn == 0.0 || j == m || iters + j >= max_iter;
                        }
                    } else if (lane == 0) {
                        s_inv = (VT)1;
                        s_stop = 0;
                    }
                }
                const int tr = (C * (r1 - r0) + 31) / 32;   // warps' worth of the finest level's rows
                if constexpr (BLK) {
                    // t = v_u - M z_w with z_w = D^-1 v_w, and the w rows of A z
                    // but for u2's part; lane pair = the two layers of a vertex
                    if (!helper)
#pragma unroll 1
                        for (int t = warp; t < tr; t += NW) {
                            const int it = t * 32 + lane, i = r0 + it / C, q = it % C, row = min(i, r1 - 1);
                            const Rows<VT> &A = tab[TAB_C];
                            const int *ce = A.c + (size_t)(row - A.base) * MGX_WT;
                            const VT *ve = A.v + (size_t)(row - A.base) * (6 * MGX_WT) + q * (3 * MGX_WT);
                            int c[MGX_WT + 2];
                            VT u[MGX_WT + 2], sm = 0, s0 = 0, s1 = 0;
#pragma unroll
                            for (int k = 0; k < MGX_WT; ++k) c[k] = NK * ce[k] + q;
                            c[MGX_WT] = NK * row + q;              // its own v_w and v_u
                            c[MGX_WT + 1] = NK * row + 2 + q;
                            ST::get(u, cw, c, ep, wt);
#pragma unroll
                            for (int k = 0; k < MGX_WT; ++k) {
                                sm += ve[k] * u[k];
                                s0 += ve[MGX_WT + k] * u[k];
                                s1 += ve[2 * MGX_WT + k] * u[k];
                            }
                            s0 += __shfl_xor_sync(0xffffffffu, s0, 1);
                            s1 += __shfl_xor_sync(0xffffffffu, s1, 1);
                            if (i < r1) {
                                const int e = NK * (i - r0) + q;
                                ST::put(c0 + (size_t)C * i + q, u[MGX_WT + 1] - sm, ep);
                                wl[e] = q ? s1 : s0;
                                wl[e + 2] = sm;
                                if (j < m) Z[(size_t)j * nk + k0 + e] = (VT)(p.dinv[k0 + e] * (double)u[MGX_WT]);
                            }
                        }
                    if (ONE) __syncthreads();
                }
                // A times T b of the finest level (and u2's part of the w2 rows)
                auto apply_tb = [&]() {
#pragma unroll 1
                    for (int t = warp; t < tr; t += NW) {
                        const int it = t * 32 + lane, i = r0 + it / C, q = it % C;
                        const Rows<VT> &A = tab[TAB_T];
                        const size_t e = (size_t)(min(i, r1 - 1) - A.base) * MGX_WT;
                        int c[MGX_WT];
                        VT u[MGX_WT], s1 = 0, s2 = 0;
#pragma unroll
                        for (int k = 0; k < MGX_WT; ++k) c[k] = C * (A.c + e)[k] + q;
                        ST::get(u, ct, c, ep, wt);
#pragma unroll
                        for (int k = 0; k < MGX_WT; ++k) {
                            s1 += (A.v2 + e)[k] * u[k];
                            if (BLK) s2 += (A.v3 + e)[k] * u[k];
                        }
                        if (i < r1) {
                            if (BLK) {
                                wl[NK * (i - r0) + 2 + q] += s1;
                                if (q) wl[NK * (i - r0) + 1] += s2;
                            } else {
                                wl[i - r0] = s1;
                            }
                        }
                    }
                };
                // down: b_{l+1} = Q_l b_l; T b of the finest level, and A times it one phase later
#pragma unroll 1
                for (int l = 0; l < bot; ++l) {
                    if (!helper) {
                        const E *src = l == 0 ? c0 : cells + p.boff[l];
                        E *dst = cells + p.boff[l + 1];
                        int i0, i1;
                        own_rows(p.x_n[l + 1], G, bi, i0, i1);
                        const int tq = ((i1 - i0) * (4 * C) + 31) / 32;  // four lanes per row of Q (and vector)
#pragma unroll 1
                        for (int t = warp; t < tq; t += NW) {
                            const int q = t * 32 + lane, i = i0 + q / (4 * C), h = (q >> 2) % C;
                            const Rows<VT> &A = tab[TAB_Q + l];
                            const size_t e = (size_t)(min(i, i1 - 1) - A.base) * MGX_WQ + (q & 3);
                            VT s = row_sum<VT, ONE, MGX_WQ / 4, 4, C>(A.c + e, A.v + e, src + h, ep, wt);
                            s += __shfl_xor_sync(0xffffffffu, s, 1);
                            s += __shfl_xor_sync(0xffffffffu, s, 2);
                            if (i < i1 && (q & 3) == 0) ST::put(dst + (size_t)C * i + h, s, ep);
                        }
                        // the finest level's rows, by the same thread in every phase
                        if (l == 0) {
#pragma unroll 1
                            for (int t = warp; t < tr; t += NW) {
                                const int it = t * 32 + lane, i = r0 + it / C, q = it % C;
                                const Rows<VT> &A = tab[TAB_T];
                                const size_t e = (size_t)(min(i, r1 - 1) - A.base) * MGX_WT;
                                const VT s = row_sum<VT, ONE, MGX_WT, 1, C>(A.c + e, A.v + e, c0 + q, ep, wt);
                                if (i < r1) {
                                    ST::put(ct + (size_t)C * i + q, s, ep);
                                    if (tl) tl[it] = s;
                                }
                            }
                        }
                        if (l == 1) apply_tb();
                    }
                    if (ONE) __syncthreads();
                }
                if (bot == 1 && !helper) apply_tb();
                // dense: x_top = [T b +] E b_bot (the first row's T b while b_bot is on its way)
                VT tb0 = 0;
                if (!helper && top > 0 && top < bot && warp < C * (d1 - d0)) {
                    const Rows<VT> &A = tab[TAB_T + top];
                    const size_t e = (size_t)(d0 + warp / C - A.base) * MGX_WT;
                    tb0 = row_sum<VT, ONE, MGX_WT, 1, C>(A.c + e, A.v + e, cells + p.boff[top] + warp % C, ep, wt);
                }
                if (!helper) {
                    const E *src = bot == 0 ? c0 : cells + p.boff[bot];
#pragma unroll 1
                    for (int q0 = warp * 32; q0 < C * nb; q0 += NW * 32) {
                        const int q = q0 + lane, c[1] = {min(q, C * nb - 1)};
                        VT t[1];
                        ST::get(t, src, c, ep, wt);
                        if (q < C * nb) bsm[(q % C) * nbs + q / C] = t[0];
                    }
                }
                if (!helper) {
                    asm volatile("bar.sync 2, %0;" ::"r"(NW * 32) : "memory");   // the workers: bsm complete
#pragma unroll 1
                    for (int t = warp; t < C * (d1 - d0); t += NW) {
                        const int i = d0 + t / C, h = t % C;
                        const VT *row = dn + (size_t)(i - d0) * nbs;
                        VT tb = 0;   // [T b] of the row
                        if (top == 0) {
                            if (bot > 0) tb = tl[i - r0];
                        } else if (top < bot && t == warp) {
                            tb = tb0;
                        } else if (top < bot) {   // level top = bot - 1
                            const Rows<VT> &A = tab[TAB_T + top];
                            const size_t e = (size_t)(i - A.base) * MGX_WT;
                            tb = row_sum<VT, ONE, MGX_WT, 1, C>(A.c + e, A.v + e, cells + p.boff[top] + h, ep, wt);
                        }
                        const VT s = dense_row<VT>(row, bsm + h * nbs, nbs, lane) + tb;
                        if (BLK || top > 0) {
                            if (lane == 0) ST::put(cells + p.xoff[top] + (size_t)C * i + h, s, ep);
                            continue;
                        }
                        VT s2 = dense_row<VT>(dn2 + (size_t)(i - d0) * nbs, bsm, nbs, lane);
                        if (lane == 0) {
                            tl[i - r0] = s;   // z and A z, not normalised yet
                            wl[i - r0] = bot > 0 ? s2 + wl[i - r0] : s2;
                        }
                    }
                }
                if (ONE) __syncthreads();
                // up: x_l = T b_l + U x_{l+1}
#pragma unroll 1
                for (int l = top - 1; l >= 1; --l) {
                    if (!helper) {
                        int i0, i1;
                        own_rows(p.x_n[l], G, bi, i0, i1);
#pragma unroll 1
                        for (int t = warp; t < (C * (i1 - i0) + 31) / 32; t += NW) {
                            const int it = t * 32 + lane, i = i0 + it / C, q = it % C, row = min(i, i1 - 1);
                            const Rows<VT> &A = tab[TAB_T + l], &U = tab[TAB_U + l];
                            const size_t e = (size_t)(row - A.base) * MGX_WT, f = (size_t)(row - U.base) * MGX_WU;
                            VT s = row_sum<VT, ONE, MGX_WT, 1, C>(A.c + e, A.v + e, cells + p.boff[l] + q, ep, wt);
                            s += row_sum<VT, ONE, MGX_WU, 1, C>(U.c + f, U.v + f, cells + p.xoff[l + 1] + q, ep, wt);
                            if (i < i1) ST::put(cells + p.xoff[l] + (size_t)C * i + q, s, ep);
                        }
                    }
                    if (ONE) __syncthreads();
                }
                // the helper's results: the stopping test and 1 / norm
                if (__syncthreads_or(s_dead)) return;
                jl = j;
                if (s_stop) break;
                const VT inv = s_inv;
                // finest level: z = T b + U x_1 and A z = A T b + A U x_1, normalised
                if (!BLK && top == 0 && !helper)
#pragma unroll 1
                    for (int q = threadIdx.x; q < kn; q += NW * 32) {
                        Z[(size_t)j * nk + k0 + q] = tl[q] * inv;
                        wl[q] *= inv;
                        vrow(j)[q] *= inv;
                    }
                if ((BLK || top > 0) && !helper)
#pragma unroll 1
                    for (int t = warp; t < tr; t += NW) {
                        const int it = t * 32 + lane, i = r0 + it / C, h = it % C, row = min(i, r1 - 1);
                        const Rows<VT> &F = tab[TAB_F];
                        const size_t e = (size_t)(row - F.base) * MGX_SF;
                        int c[MGX_WF];
                        VT tb[1], x1[MGX_WF];
#pragma unroll
                        for (int q = 0; q < MGX_WF; ++q) c[q] = C * (F.c + e)[q] + h;
                        if (tl) {
                            tb[0] = tl[min(it, C * (r1 - r0) - 1)];
                        } else {   // this block's own T b
                            const int ci[1] = {C * row + h};
                            ST::get(tb, ct, ci, ep, wt);
                        }
                        ST::get(x1, cells + p.xoff[1], c, ep, wt);
                        VT s = 0, aw = 0, ew = 0;
#pragma unroll
                        for (int q = 0; q < MGX_WF; ++q) {
                            s += (F.v + e)[q] * x1[q];
                            aw += (F.v2 + e)[q] * x1[q];
                            if (BLK) ew += (F.v3 + e)[q] * x1[q];
                        }
                        if (i < r1) {
                            const int q = NK * (i - r0) + h;
                            VT *vj = vrow(j), *zj = Z + (size_t)j * nk + k0;
                            if (BLK) {
                                zj[q] *= inv;
                                zj[q + 2] = -(tb[0] + s) * inv;
                                wl[q] = (h ? wl[q] + ew : wl[q]) * inv;
                                wl[q + 2] = (wl[q + 2] + aw) * inv;
                                vj[q] *= inv;
                                vj[q + 2] *= inv;
                            } else {
                                zj[q] = (tb[0] + s) * inv;
                                wl[q] = (wl[q] + aw) * inv;
                                vj[q] *= inv;
                            }
                        }
                    }
                if (BLK) __syncthreads();   // the vectors' entries change hands
                my_cols += j + 1;
                // dots with v_0..v_j, eight basis vectors per pass, on this thread's own rows
                if (warp < NA)
#pragma unroll 1
                    for (int l0 = 0; l0 <= j; l0 += 8) {
                        VT t[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                        const int kk = min(8, j + 1 - l0);
                        if (l0 + 8 <= p.mvp) {   // all in shared memory (those past j: not used)
                            const VT *v0 = vsm + l0 * rpb;
#pragma unroll 1
                            for (int q = threadIdx.x; q < kn; q += NW * 32) {
                                const VT s = wl[q];
#pragma unroll
                                for (int k = 0; k < 8; ++k) t[k] += v0[k * rpb + q] * s;
                            }
                        } else {
                            const VT *vp[8];
#pragma unroll
                            for (int k = 0; k < 8; ++k) vp[k] = vrow(l0 + (k < kk ? k : 0));
#pragma unroll 1
                            for (int q = threadIdx.x; q < kn; q += NW * 32) {
                                const VT s = wl[q];
#pragma unroll
                                for (int k = 0; k < 8; ++k) t[k] += vp[k][q] * s;
                            }
                        }
                        const VT s = fold8(t, lane);
                        const int k = lane >> 2;   // bits 4, 3, 2 of the lane: value 4 h16 + 2 h8 + h4
                        if ((lane & 3) == 0 && k < kk) redv[(l0 + k) * RS + warp] = s;
                    }
                __syncthreads();
#pragma unroll 1
                for (int l = warp; l <= j; l += NW + 1) {
                    double s = lane < NA ? (double)redv[l * RS + lane] : 0.0;
                    s = lanes_sum(s, NA);
                    const VT q = (VT)s;
                    if constexpr (ONE) {
                        if (lane == 0) { hcol[l] = (double)q; hv[l] = q; }
                    } else {
                        E *dp = cpart + (size_t)l * G;
                        if (lane == 0) ST::put(dp + bi, q, ep);
                        if (bi == l % G) {
                            const VT t = root_sum<VT>(dp, G, ep, wt);
                            if (lane == 0) ST::put(csum + l, t, ep);
                        }
                    }
                }
                if constexpr (!ONE)
                    if (helper) {
                        const int c[2] = {min(lane, j), min(lane + 32, j)};
                        VT t[2];
                        ST::get(t, csum, c, ep, wt);
                        if (lane <= j) { hcol[lane] = (double)t[0]; hv[lane] = t[0]; }
                        if (lane + 32 <= j) { hcol[lane + 32] = (double)t[1]; hv[lane + 32] = t[1]; }
                    }
                if (__syncthreads_or(s_dead)) return;
                if (helper) {
                    if (lane == 0) {   // the earlier rotations on the new column
                        double a = hcol[0];
#pragma unroll 1
                        for (int l = 0; l < j; ++l) {
                            const double c = hcol[l + 1];
                            H[l * MAXM + j] = cs[l] * a + sn[l] * c;
                            a = -sn[l] * a + cs[l] * c;
                        }
                        s_a = a;
                    }
                } else {
                    // w -= sum h_l v_l, and its norm's partial sum
                    VT a2 = 0;
                    VT *vn = vrow(j + 1);
#pragma unroll 1
                    for (int q = threadIdx.x; q < kn; q += NW * 32) {
                        VT s = wl[q];
#pragma unroll 1
                        for (int l0 = 0; l0 <= j; l0 += 8) {
                            const int kk = min(8, j + 1 - l0);
                            if (l0 + 8 <= p.mvp) {
                                const VT *v0 = vsm + l0 * rpb + q;
#pragma unroll
                                for (int k = 0; k < 8; ++k)
                                    if (k < kk) s -= hv[l0 + k] * v0[k * rpb];
                            } else {
                                VT vq[8];
#pragma unroll
                                for (int k = 0; k < 8; ++k) vq[k] = vrow(l0 + (k < kk ? k : 0))[q];
#pragma unroll
                                for (int k = 0; k < 8; ++k)
                                    if (k < kk) s -= hv[l0 + k] * vq[k];
                            }
                        }
                        vn[q] = s;
                        ST::put(cw + k0 + q, s, ep + 1);
                        a2 += s * s;
                    }
                    if (warp < NA) {
                        a2 = warp_sum(a2);
                        if (lane == 0) redv[warp] = a2;
                    }
                    if (!ONE) asm volatile("bar.arrive 1, %0;" ::"r"((int)blockDim.x) : "memory");
                }
                if (ONE) __syncthreads();
            }
            iters += jl;
            my_steps += jl;
            // y = H^-1 g (reciprocal diagonal in parallel, then column by
            // column) and x += sum_l y_l z_l, formed in the Krylov precision
            // and added to the FP64 iterate once
            if (warp == 0) {
#pragma unroll 1
                for (int l = lane; l < jl; l += 32) y[l] = 1.0 / H[l * MAXM + l];
                __syncwarp();
#pragma unroll 1
                for (int l = jl - 1; l >= 0; --l) {
                    const double yl = g[l] * y[l];
                    __syncwarp();
                    if (lane == 0) y[l] = yl;
#pragma unroll 1
                    for (int k = lane; k < l; k += 32) g[k] -= H[k * MAXM + l] * yl;
                    __syncwarp();
                }
#pragma unroll 1
                for (int l = lane; l < jl; l += 32) hv[l] = (VT)y[l];
            }
            __syncthreads();
            if (!helper)
#pragma unroll 1
                for (int i = k0 + threadIdx.x; i < k0 + kn; i += NW * 32) {
                    VT s = 0;
#pragma unroll 8
                    for (int l = 0; l < jl; ++l) s += hv[l] * Z[(size_t)l * nk + i];
                    x[i] += (double)s;
                }
            if (!group_sync(bar, G, err, nullptr)) return;   // x complete
        }
        my_iters = max(my_iters, iters);
        my_cycles = max(my_cycles, cycles);
        // the next right-hand side reuses the cells and the shared memory
        if (v + p.groups < p.nv && !group_sync(bar, G, err, nullptr)) return;
    }
    if (threadIdx.x == 0)
        atomicAdd(&p.stats->bytes, (double)kn * (my_resid * p.resid_row_bytes + my_steps * (p.step_row_bytes + es) +
                                                 2.0 * es * my_cols + 24.0 * my_cycles));
    if (threadIdx.x == 0 && bi == 0) {
        atomicAdd(&p.stats->steps_total, my_steps);
        atomicMax(&p.stats->iters, my_iters);
        atomicMax(&p.stats->cycles, my_cycles);
        atomicMax(&p.stats->status, my_status);
        // relres >= 0: max via the integer order of non-negative doubles
        atomicMax((unsigned long long *)&p.stats->relres, (unsigned long long)__double_as_longlong(my_rel));
    }
}

size_t mgs_fixed_smem() {
    return sizeof(double) * ((MAXM + 1) * MAXM + 2 * MAXM + (MAXM + 1) + MAXM + (MAXM + 2) + (MAXM + 2) * RS) +
           sizeof(double) * (MAXM + 2);
}

void *mgs_fn(Precision prec, int kind) {   // kind 0: blocks share right-hand sides, 1: a block each, 2: block system
    if (prec == PREC_MIXED)
        return kind == 0 ? (void *)mgs_kernel<float, false, false>
             : kind == 1 ? (void *)mgs_kernel<float, true, false> : (void *)mgs_kernel<float, false, true>;
    return kind == 0 ? (void *)mgs_kernel<double, false, false>
         : kind == 1 ? (void *)mgs_kernel<double, true, false> : (void *)mgs_kernel<double, false, true>;
}

// bytes of dynamic shared memory a block may take (set once per kernel)
cudaError_t mgs_smem_limit(Precision prec, int kind, int *limit) {
    static std::once_flag once[6];
    static cudaError_t err[6];
    static int lim[6];
    const int k = (prec == PREC_MIXED ? 1 : 0) + 2 * kind;
    std::call_once(once[k], [&] {
        int dev = 0, optin = 0;
        cudaFuncAttributes fa;
        if ((err[k] = cudaGetDevice(&dev)) != cudaSuccess) return;
        if ((err[k] = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess) return;
        if ((err[k] = cudaFuncGetAttributes(&fa, mgs_fn(prec, kind))) != cudaSuccess) return;
        lim[k] = optin - (int)fa.sharedSizeBytes;
        err[k] = cudaFuncSetAttribute(mgs_fn(prec, kind), cudaFuncAttributeMaxDynamicSharedMemorySize, lim[k]);
    });
    *limit = lim[k];
    return err[k];
}

}  // namespace

size_t mgs_scratch_bytes(const DevSolveOp &op, Precision prec) {
    const size_t cell = prec == PREC_MIXED ? 8 : 16;
    const size_t C = op.block4 ? 2 : 1, n = (size_t)op.mgx.lev[0].n;
    size_t cells = op.block4 ? 8 * n : 2 * n;
    for (int l = 1; l < op.mgx.nlev; ++l) cells += 2 * C * op.mgx.lev[l].n;
    return (cells * cell + 255) & ~size_t(255);
}

bool mgs_applicable(const DevSolveOp &op) {
    return op.mgx.nlev >= 2 && (op.block4 ? op.blk.c != nullptr : op.A.W <= 8);
}

cudaError_t mgs_prepare() {
    int lim;
    cudaError_t e = cudaSuccess;
    for (Precision prec : {PREC_FP64, PREC_MIXED})
        for (int kind = 0; kind < 3 && e == cudaSuccess; ++kind) e = mgs_smem_limit(prec, kind, &lim);
    return e;
}

cudaError_t mgs_solve(const DevSolveOp &op, const MgsArgs &q, cudaStream_t s) {
    const MgxDev &x = op.mgx;
    const bool blk = op.block4 != 0;
    const size_t C = blk ? 2 : 1, NK = blk ? 4 : 1;
    const int n = x.lev[0].n, nlev = x.nlev;
    const bool mixed = q.prec == PREC_MIXED;
    const size_t es = mixed ? 4 : 8;
    const int sms = (q.max_sms > 0 && q.max_sms < q.sms) ? q.max_sms : q.sms;
    // One block per SM with all its shared memory, its warps split over the
    // rows; two smaller blocks per SM where that spreads the right-hand sides
    // better: more of them than SMs, or more than half as many but few enough
    // for three blocks each (level 5, 100 FP64 right-hand sides: 6.4 ms with one
    // block each on 100 of 152 SMs, 4.3 ms with three half-size blocks; level 4,
    // 152 mixed ones: 0.92 ms with one block, 1.20 ms with two halves).
    // Two smaller blocks also where the caller leaves this launch a part of the
    // SMs: others run beside it, and an SM seldom empties for a block that
    // needs all of it.
    const bool half = sms < q.sms || q.nv > sms || (2 * q.nv > sms && 2 * sms / q.nv >= 3);
    int workers = half ? 256 : (mixed ? 768 : 512);
    const int cap = half ? 2 * sms : sms;
    const int groups = std::min(q.nv, cap);
    int G = cap / groups;
    if (q.rpb > 0) G = std::min(G, (n + q.rpb - 1) / q.rpb);
    G = std::max(G, 1);
    const bool one = G == 1 && !blk;
    int limit = 0;
    cudaError_t e = mgs_smem_limit(q.prec, blk ? 2 : one ? 1 : 0, &limit);
    if (e != cudaSuccess) return e;
    size_t budget = (size_t)limit;
    if (half) budget = std::min<size_t>(budget, 104 * 1024);

    MgsParams p;
    memset(&p, 0, sizeof p);
    for (int l = 0; l < nlev; ++l) p.x_n[l] = x.lev[l].n;
    // Where the dense product starts.  Each sparse level costs two hand-overs
    // (about 1,500 cycles each between blocks, 150 within one); a dense product
    // costs its multiply-adds per block, taken at 48 FP32 or 1.6 FP64 a cycle from
    // shared memory and 14 or 1.5 from L2.  Against every start forced in turn
    // (noise, to 1e-12; 1, 8, 37 and 160 right-hand sides on levels 3 to 5, 1 and 8
    // on 6 and 7, both precisions) the choice is within 3 % of the
    // best in 27 of 31 cases; one FP64 solve on level 3 249 us with it and 233 with
    // the finest level dense, and one or two levels further down would be 9 to 15 %
    // faster for 8 and 37 mixed ones on level 5 (37: 1,193 and 1,040 us) and 8 FP64
    // ones on level 6.
    double best = 1e300;
    for (int k = x.first_dense; k < nlev; ++k)
        for (int wide = 0; wide < 2; ++wide) {
            const int top = k - wide;
            if (wide && (k != x.first_dense || !x.E)) continue;
            if (top == 0 && (blk || !(wide ? x.AE : x.AB))) continue;
            const double rows = (double)((x.lev[top].n + G - 1) / G), ent = rows * x.lev[k].n * (top == 0 ? 2.0 : 1.0);
            const bool cached = mgs_fixed_smem() + es * ent < 0.6 * (double)budget;
            const double rate = mixed ? (cached ? 48.0 : 14.0) : (cached ? 1.6 : 1.5);
            const int hand = (k > 0 ? k : 0) + (top > 0 ? top : 0);
            const double cost = hand * (one ? 150.0 : 1500.0) + ent / rate * (half ? 2.0 : 1.0);
            if (cost < best) { best = cost; p.top = top; p.bot = k; }
        }
    // shared memory: the coarse levels' rows, the dense rows, then the finest
    // level's and as many Krylov vectors as fit
    size_t used = (mgs_fixed_smem() + 15) & ~size_t(15);
    auto take = [&](size_t bytes) -> int {
        bytes = (bytes + 15) & ~size_t(15);
        if (used + bytes > budget) return -1;
        const int o = (int)used;
        used += bytes;
        return o;
    };
    auto rpb = [&](int l) { return (size_t)((x.lev[l].n + G - 1) / G); };
    p.off_b = take(C * es * (size_t)mgx_stride(x.lev[p.bot].n));
    if (p.off_b < 0) return cudaErrorInvalidValue;
    p.off_w = take(NK * es * rpb(0));
    p.off_t = take(C * es * rpb(0));
    auto copy = [&](const void *src, int rows, int words, int dst) {
        Copy &c = p.copy[p.ncopy++];
        c.src = src; c.rows = rows; c.words = words; c.dst = dst;
    };
    // one to three value arrays of vw values a row on a pattern of `width` entries
    auto table = [&](int t, const int *c, const void *v, const void *v2, const void *v3, int rows, size_t rows_b,
                     int width, int vw) {
        Table &T = p.tab[t];
        T.c = c; T.v = v; T.v2 = v2; T.v3 = v3; T.rows = rows;
        const size_t vb = (rows_b * vw * es + 15) & ~size_t(15);
        const int arrays = v3 ? 3 : v2 ? 2 : 1;
        T.off = take(arrays * vb + rows_b * width * 4);
        if (T.off < 0) return;
        T.off2 = T.off + (int)vb;
        T.off3 = T.off2 + (int)vb;
        T.offc = T.off + arrays * (int)vb;
        copy(v, rows, vw * (int)es / 4, T.off);
        if (v2) copy(v2, rows, vw * (int)es / 4, T.off2);
        if (v3) copy(v3, rows, vw * (int)es / 4, T.off3);
        copy(c, rows, width, T.offc);
    };
    for (int t = 0; t < N_TAB; ++t) p.tab[t].off = -1;
    for (int l = p.bot - 1; l >= 1; --l) {
        table(TAB_T + l, x.lev[l].tc, x.lev[l].tv, nullptr, nullptr, x.lev[l].n, rpb(l), MGX_WT, MGX_WT);
        table(TAB_Q + l, x.lev[l].qc, x.lev[l].qv, nullptr, nullptr, x.lev[l + 1].n, rpb(l + 1), MGX_WQ, MGX_WQ);
        if (l < p.top)
            table(TAB_U + l, x.lev[l].uc, x.lev[l].uv, nullptr, nullptr, x.lev[l].n, rpb(l), MGX_WU, MGX_WU);
    }
    p.dense = p.top < p.bot ? x.E : x.B[p.bot];
    p.dense2 = p.top == 0 ? (p.bot == 0 ? x.AB : x.AE) : nullptr;
    {
        const int stride = mgx_stride(x.lev[p.bot].n);
        const size_t db = es * rpb(p.top) * stride;
        p.off_d = take(db * (p.top == 0 ? 2 : 1));
        p.off_d2 = p.off_d + (int)db;
        if (p.off_d >= 0) {
            copy(p.dense, x.lev[p.top].n, stride * (int)es / 4, p.off_d);
            if (p.dense2) copy(p.dense2, x.lev[p.top].n, stride * (int)es / 4, p.off_d2);
        }
    }
    if (p.bot > 0) {
        table(TAB_T, x.lev[0].tc, x.lev[0].tv, x.a, blk ? op.blk.e4 : nullptr, n, rpb(0), MGX_WT, MGX_WT);
        table(TAB_Q, x.lev[0].qc, x.lev[0].qv, nullptr, nullptr, x.lev[1].n, rpb(1), MGX_WQ, MGX_WQ);
    }
    if (p.top > 0) table(TAB_F, x.fc, x.fu, x.fa, blk ? op.blk.e4u : nullptr, n, rpb(0), MGX_SF, MGX_SF);
    if (blk) table(TAB_C, op.blk.c, op.blk.v, nullptr, nullptr, n, rpb(0), MGX_WT, 6 * MGX_WT);
    p.off_v = (int)used;
    // whole batches of eight, also past the last vector
    p.mvp = (int)std::min<size_t>((q.m + 8) / 8 * 8, (budget - used) / (NK * es * rpb(0)) / 8 * 8);
    p.mv = std::min(p.mvp, q.m + 1);
    used += (size_t)p.mvp * NK * es * rpb(0);

    p.col = op.A.col; p.aval = op.A.val; p.dinv = op.dinv;
    p.W = op.A.W; p.n = n; p.nv = q.nv; p.ld = q.ld; p.m = q.m; p.max_iter = q.max_iter;
    p.tol = q.tol; p.inner_rtol = q.inner_rtol;
    p.B = q.B; p.X = q.X;
    p.V = q.V; p.Z = q.Z; p.Wv = q.Wv; p.R = q.R;
    p.scratch = q.scratch;
    p.group_bytes = mgs_scratch_bytes(op, q.prec);
    p.part = q.part;
    // the stamped sums behind the plain ones: 2 (MAXM + 2) doubles a block each
    p.cpart = (char *)(q.part + (size_t)groups * G * 2 * (MAXM + 2));
    p.bar = q.bar; p.err = &q.stats->status; p.stats = q.stats;
    p.groups = groups; p.G = G;
    p.wait_limit = q.wait_limit;
    size_t c = (blk ? 8 : 2) * (size_t)n;
    for (int l = 1; l < nlev; ++l) { p.boff[l] = c; c += C * x.lev[l].n; p.xoff[l] = c; c += C * x.lev[l].n; }
    // algorithmic bytes per finest row: the residual, and one Arnoldi step
    // (operators once, each level's vectors once in and once out, w and v)
    p.resid_row_bytes = op.A.W * 12.0 + 24.0;
    p.step_row_bytes = 6.0 * es;
    for (int l = 0; l < p.bot; ++l) {
        const double f = (double)x.lev[l].n / n, fc = (double)x.lev[l + 1].n / n;
        p.step_row_bytes += f * (MGX_WT * (4.0 + es) + 2.0 * es) + fc * (MGX_WQ * (4.0 + es) + 2.0 * es);
        if (l >= 1 && l < p.top) p.step_row_bytes += f * MGX_WU * (4.0 + es);
    }
    if (p.bot > 0) p.step_row_bytes += op.A.W * es;
    if (p.top > 0) p.step_row_bytes += MGX_WF * (4.0 + 2.0 * es);
    p.step_row_bytes += (double)x.lev[p.top].n * x.lev[p.bot].n * es / n * (p.top == 0 ? 2.0 : 1.0);
    // per Krylov entry of a block system: four per finest row, the matrices read once for both vectors
    if (blk) p.step_row_bytes = p.step_row_bytes / 4.0 + 7.0 * (4.0 + 6.0 * es) / 4.0 + 6.0 * es;

    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute coop[1];
    coop[0].id = cudaLaunchAttributeCooperative;
    coop[0].val.cooperative = 1;
    cfg.gridDim = dim3(groups * G);
    cfg.blockDim = dim3(workers + 32);
    cfg.dynamicSmemBytes = used;
    cfg.stream = s;
    cfg.attrs = coop;
    cfg.numAttrs = 1;
    void *args[] = {&p};
    if ((e = cudaLaunchKernelExC(&cfg, mgs_fn(q.prec, blk ? 2 : one ? 1 : 0), args)) != cudaSuccess) return e;
    ++g_kernel_launches;
    return cudaGetLastError();
}

}  // namespace phg
