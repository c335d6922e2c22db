// The stamped cells' waits (phg_stamp.cuh) outside a solver: one launch of two
// groups of two blocks.  Block 0 of a group waits for a cell that nobody
// writes, block 1 waits for block 0 at the group's barrier.  Group 0 has a
// limit of LIMIT cycles, group 1 one of LONG: when group 0 gives up, group 1
// has to leave for the launch's error flag, at the cell and at the barrier.
#include <cstdio>

#include "phg_stamp.cuh"

using namespace phg;

constexpr long long LIMIT = 2000000, LONG = 2000000000;

struct Result { long long cycles; int dead, passed; double value; };

template <typename VT>
__global__ void waits(Cell<VT> *cells, unsigned *bar, int *err, Result *res) {
    __shared__ int dead;
    __shared__ long long since[2];
    const int grp = blockIdx.x / 2, bi = blockIdx.x % 2;
    const long long limit = grp == 0 ? LIMIT : LONG;
    if (threadIdx.x == 0) {
        wait_limit_slot() = limit;
        bar_epoch() = 0;
        dead = 0;
    }
    __syncthreads();
    const Waits w = {err, (unsigned long long *)(bar + 2 * grp), &dead, since, limit};
    const long long t0 = clock64();
    int passed = 1;
    VT x[2] = {0, 0};
    if (bi == 0) {
        const int there[2] = {0, 1}, never[2] = {0, 2};
        wait_cells<VT, 2>(x, cells, there, 1u, w);           // both carry the stamp 1
        if (dead) x[0] = x[1] = 0;
        VT y[2];
        wait_cells<VT, 2>(y, cells, never, 1u, w);           // cell 2 never does
        passed = !__syncthreads_or(dead);
    } else {
        passed = group_sync(bar + 2 * grp, 2, err, nullptr);
    }
    if (threadIdx.x == 0) res[blockIdx.x] = Result{clock64() - t0, dead, passed, (double)(x[0] + x[1])};
}

template <typename VT> __global__ void put(Cell<VT> *cells) {
    st_cell(cells, (VT)1.5, 1u);
    st_cell(cells + 1, (VT)2.25, 1u);
    st_cell(cells + 2, (VT)0, 0u);
}

#define CK(call) do { cudaError_t e = (call); if (e != cudaSuccess) { printf("%s: %s\n", #call, cudaGetErrorString(e)); return 1; } } while (0)

template <typename VT> int run(const char *name) {
    Cell<VT> *cells;
    unsigned *bar;
    int *err, flag = 0, bad = 0;
    Result *res, h[4];
    CK(cudaMalloc(&cells, 3 * sizeof(Cell<VT>)));
    CK(cudaMalloc(&bar, 4 * sizeof(unsigned)));
    CK(cudaMalloc(&err, sizeof(int)));
    CK(cudaMalloc(&res, sizeof h));
    CK(cudaMemset(bar, 0, 4 * sizeof(unsigned)));
    CK(cudaMemset(err, 0, sizeof(int)));
    put<VT><<<1, 1>>>(cells);
    void *args[] = {&cells, &bar, &err, &res};
    CK(cudaLaunchCooperativeKernel((void *)waits<VT>, dim3(4), dim3(64), args, 0, 0));
    CK(cudaDeviceSynchronize());
    CK(cudaMemcpy(h, res, sizeof h, cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(&flag, err, sizeof flag, cudaMemcpyDeviceToHost));
    bad |= flag != STATUS_TIMEOUT;
    for (int b = 0; b < 4; ++b) {
        printf("%s block %d: %lld cycles, dead %d, passed %d, value %g\n", name, b, h[b].cycles, h[b].dead, h[b].passed,
               h[b].value);
        bad |= h[b].passed;
        // the limit, and 2 x 64 loads, another 64 until group 1 sees the flag, at no more than 5,000 cycles each
        bad |= h[b].cycles > LIMIT + 192 * 5000;
        if (b % 2 == 0) bad |= !h[b].dead || h[b].value != 3.75;
    }
    bad |= h[0].cycles < LIMIT;
    return bad;
}

int main() {
    if (run<float>("fp32") || run<double>("fp64")) return 1;
    printf("waits ended\n");
    return 0;
}
