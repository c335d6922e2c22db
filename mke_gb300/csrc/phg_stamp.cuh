// phg_stamp.cuh -- values that carry their own ready mark.
//
// A persistent solver's phases hand values from block to block: each row
// gathers its neighbours' results of the phase before.  A group barrier
// between two phases costs about 3,000 cycles on this part (drain the stores,
// one reduction and one poll at L2, an L1 invalidation: measured 2,955 with
// 152 blocks), the phase itself a few hundred.  Here a value and the number of
// the phase that wrote it ("stamp") sit in one word that is read and written
// in one piece (64 bits for FP32, 128 for FP64), and a reader repeats its load
// until the stamp is the one it needs: no barrier and no fence, about 1,500
// (FP32) and 2,000 (FP64) cycles per phase, measured with 7 gathers per row
// and 152 blocks.
//
// A cell may be rewritten only when every reader of its old value is known to
// have read it; each user of these functions says why that holds.
//
// The lanes of a warp read together and go on together (a loop per lane would
// let lanes that wait block lanes that have to write).  Every wait is bounded: a
// warp looks at the clock at every 64th load, and once it has waited for the
// launch's limit (beyond the first 64 loads) it raises the launch's error flag.
// A warp that gives up, for its own limit or for the flag, poisons its group's
// barrier word, so that no block of the group waits there for its block, and
// marks its block, whose other warps stop waiting too and whose next
// __syncthreads leads out of the kernel.
#pragma once
#include "phg_group.cuh"

namespace phg {

namespace {

template <typename VT> struct CellOf;
template <> struct CellOf<float> { using T = unsigned long long; };
template <> struct CellOf<double> { using T = ulonglong2; };
template <typename VT> using Cell = typename CellOf<VT>::T;

// (No memory clobber: the stamp is the only order a cell's value needs, and the
// loads of matrix entries may move across the waits.)
__device__ __forceinline__ void st_cell(unsigned long long *p, float v, unsigned stamp) {
    const unsigned long long w = ((unsigned long long)stamp << 32) | __float_as_uint(v);
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(w));
}
__device__ __forceinline__ void ld_cell(const unsigned long long *p, float &v, unsigned &stamp) {
    unsigned long long w;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(w) : "l"(p));
    v = __uint_as_float((unsigned)w);
    stamp = (unsigned)(w >> 32);
}
__device__ __forceinline__ void st_cell(ulonglong2 *p, double v, unsigned stamp) {
    asm volatile("{.reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t;}" ::"l"(p),
                 "l"(__double_as_longlong(v)), "l"((unsigned long long)stamp));
}
__device__ __forceinline__ void ld_cell(const ulonglong2 *p, double &v, unsigned &stamp) {
    unsigned long long a, b;
    asm volatile("{.reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t;}"
                 : "=l"(a), "=l"(b)
                 : "l"(p));
    v = __longlong_as_double((long long)a);
    stamp = (unsigned)b;
}

// what a waiting warp needs to give up
struct Waits {
    int *err;                   // the launch's error flag (the status of its record)
    unsigned long long *bar;    // the group's barrier word
    int *dead;                  // shared: this block gives up
    long long *since;           // shared, one per warp: when its wait began (a register would be held through every wait)
    long long limit;            // clock cycles that a wait may take
};

// x[q] = the value of cell p[c[q]] once all N of every lane carry `stamp`.
// All 32 lanes call it together.
template <typename VT, int N>
__device__ __forceinline__ void wait_cells(VT (&x)[N], const Cell<VT> *p, const int (&c)[N], unsigned stamp,
                                           const Waits &w) {
#pragma unroll 1
    for (unsigned round = 0;; ++round) {
        unsigned e[N], miss = 0;
#pragma unroll
        for (int q = 0; q < N; ++q) ld_cell(p + c[q], x[q], e[q]);
#pragma unroll
        for (int q = 0; q < N; ++q) miss |= e[q] ^ stamp;
        if (!__any_sync(0xffffffffu, miss != 0)) return;
        if ((round & 63u) == 63u) {   // inline: a call here would put a register save at every wait
            volatile long long *since = w.since + (threadIdx.x >> 5);
            if (round == 63u) *since = clock64();
            const bool late = clock64() - *since > w.limit;
            if (__any_sync(0xffffffffu, late || *(volatile int *)w.dead || *(volatile int *)w.err == STATUS_TIMEOUT)) {
                if (late) atomicMax(w.err, STATUS_TIMEOUT);
                atomicOr(w.bar, BAR_POISON);
                *(volatile int *)w.dead = 1;
                return;
            }
        }
    }
}

// A vector whose elements are handed from block to block (stamped cells), or,
// when one block owns every row (ONE), plain values ordered by __syncthreads.
template <typename VT, bool ONE> struct CellStore;
template <typename VT> struct CellStore<VT, true> {
    using E = VT;
    __device__ static void put(E *p, VT v, unsigned) { *p = v; }
    template <int N>
    __device__ static void get(VT (&x)[N], const E *p, const int (&c)[N], unsigned, const Waits &) {
#pragma unroll
        for (int q = 0; q < N; ++q) x[q] = p[c[q]];
    }
    __device__ static VT own(const E *p) { return *p; }
};
template <typename VT> struct CellStore<VT, false> {
    using E = Cell<VT>;
    __device__ static void put(E *p, VT v, unsigned stamp) { st_cell(p, v, stamp); }
    template <int N>
    __device__ static void get(VT (&x)[N], const E *p, const int (&c)[N], unsigned stamp, const Waits &w) {
        wait_cells<VT, N>(x, p, c, stamp, w);
    }
    __device__ static VT own(const E *p) {   // written by this block before its last __syncthreads
        VT v;
        unsigned e;
        ld_cell(p, v, e);
        return v;
    }
};

}  // namespace

}  // namespace phg
