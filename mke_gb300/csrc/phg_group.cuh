// phg_group.cuh -- the barrier between the blocks of one group of a persistent
// solver launch, and the small device helpers the solver kernels share.
#pragma once
#include <cuda_runtime.h>

namespace phg {

constexpr int MAXM = 48;         // largest restart length
constexpr int STATUS_TIMEOUT = 2;  // GmresStats::status of a launch that gave up a wait (also its error flag)
constexpr long long SPIN_LIMIT = 2000000000LL;  // default wait limit, clock64 cycles (~1 s)

// phase cycle counters kept by block 0 when PHG_PHASE_TIMING is set
enum { T_RESID, T_VCYCLE, T_SPMV_DOT, T_DOT_SUM, T_UPDATE, T_NORM_SUM, T_GIVENS, T_CORR, T_BARRIER,
       T_BARRIERS, T_TOTAL, T_NPHASE };

namespace {

// The launch's barrier wait limit, held by thread 0 of every block (the only
// thread that waits): set once at kernel entry.
__device__ __forceinline__ long long &wait_limit_slot() {
    __shared__ long long lim;
    return lim;
}

// Barriers this block has passed in the launch, held by thread 0 (set to 0 at
// kernel entry, with the wait limit).
__device__ __forceinline__ unsigned long long &bar_epoch() {
    __shared__ unsigned long long e;
    return e;
}

constexpr unsigned long long BAR_POISON = 1ull << 62;

__device__ __forceinline__ unsigned long long ld_relaxed(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// Barrier of the G blocks of one group; false if the group is aborting.  The
// group's 64-bit word at bar counts arrivals and is never reset within a
// launch (nor wraps).  Every block of a group passes the same sequence of
// barriers, so at its k-th barrier (k from 1) a block adds one and waits until
// the count reaches k * G: the last arrival releases everyone (no reset, no
// second flag), and a block that runs ahead into the next barrier only raises
// the count further.  The arrival is a release reduction that returns nothing.
//
// What bounds it: round trips to L2 by one thread.  The wait therefore reads
// one word only -- a block that gives up (after the launch's wait limit) sets
// the word's poison bit, which ends every later wait of the group as well, so
// no separate error flag is read on the way -- with relaxed loads, and one
// fence after the last of them instead of an acquire on each.
__device__ bool group_sync(unsigned *bar, int G, int *err, long long *tm) {
    __shared__ int ok;
    long long tb = (tm && threadIdx.x == 0) ? clock64() : 0;
    __syncthreads();
    if (G == 1) return true;   // nothing to wait for
    if (threadIdx.x == 0) {
        unsigned long long *cnt = reinterpret_cast<unsigned long long *>(bar);   // 8-byte aligned
        const unsigned long long target = ++bar_epoch() * (unsigned long long)G;
        // release: the block's writes (ordered before this thread by the
        // __syncthreads above) are visible device-wide before the arrival
        asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(cnt) : "memory");
        const long long t0 = clock64(), lim = wait_limit_slot();
        unsigned long long v;
        while ((v = ld_relaxed(cnt)) < target) {   // the poison bit is above any target
            if (clock64() - t0 > lim) {
                atomicOr(cnt, BAR_POISON);
                atomicMax(err, STATUS_TIMEOUT);
                v = BAR_POISON;
                break;
            }
        }
        // acquire: the load that saw the count completes before any later
        // access of the block (the __syncthreads below orders the others)
        asm volatile("fence.acq_rel.gpu;" ::: "memory");
        ok = v < BAR_POISON;
        if (tm) { tm[T_BARRIER] += clock64() - tb; tm[T_BARRIERS]++; }
    }
    __syncthreads();
    return ok;
}

template <typename T> __device__ __forceinline__ T ldcg(const T *p) { return __ldcg(p); }

__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ float warp_sum(float v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// the warp's sums of eight values per lane with 9 additions instead of 40:
// halves exchange four, two and one of them, then two plain steps; lane l
// returns the sum of value (l >> 2) & 7 (bit-reversed pairs, see the caller)
template <typename T>
__device__ __forceinline__ T fold8(const T (&t)[8], int lane) {
    T a[4], b[2];
    const bool h16 = lane & 16, h8 = lane & 8, h4 = lane & 4;
#pragma unroll
    for (int k = 0; k < 4; ++k) a[k] = (h16 ? t[k + 4] : t[k]) + __shfl_xor_sync(0xffffffffu, h16 ? t[k] : t[k + 4], 16);
#pragma unroll
    for (int k = 0; k < 2; ++k) b[k] = (h8 ? a[k + 2] : a[k]) + __shfl_xor_sync(0xffffffffu, h8 ? a[k] : a[k + 2], 8);
    T c = (h4 ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, h4 ? b[0] : b[1], 4);
    c += __shfl_xor_sync(0xffffffffu, c, 2);
    c += __shfl_xor_sync(0xffffffffu, c, 1);
    return c;   // value 4 (lane >> 4 & 1) + 2 (lane >> 3 & 1) + (lane >> 2 & 1)
}

// sum over the first `na` lanes (a power-of-two tree no larger than needed), in every lane
__device__ __forceinline__ double lanes_sum(double v, int na) {
    for (int o = 1; o < na; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return __shfl_sync(0xffffffffu, v, 0);
}

// maximum that keeps a NaN (fmax drops it): a non-finite residual must reach
// the host as such, never as the other operand
__device__ __forceinline__ double max_nan(double a, double b) { return a != a ? a : (b != b ? b : fmax(a, b)); }

// rows [r0, r1) of a level of size n split over G blocks
__device__ __forceinline__ void own_rows(int n, int G, int bi, int &r0, int &r1) {
    const int rpb = (n + G - 1) / G;
    r0 = min(n, bi * rpb);
    r1 = min(n, r0 + rpb);
}

}  // namespace

}  // namespace phg
