// Waits that run out: a barrier that nothing arrives at, with a short limit (see test_gpu_waits.py).
#define SMLA_LEAN_POLLS 4096u
#include "sm100_ptx.cuh"

using namespace smla::ptx;

// result: [0] a wait for a phase that completes, [1] and [2] two that never do, one after the other, [3] the code on record
__global__ void wait_kernel(int* result, long long* cycles) {
    __shared__ alignas(8) unsigned long long bars[2];
    __shared__ int flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t done = smem_u32(&bars[0]), never = smem_u32(&bars[1]), flag_addr = smem_u32(&flag);
    if (threadIdx.x == 0) {
        mbar_init(done, 1);
        mbar_init(never, 1);
        flag = 0;
        mbar_init_fence();
        mbar_arrive(done);
    }
    __syncthreads();
    for (int turn = 0; turn < 3; ++turn) {
        if (warp == turn) {
            const long long t0 = clock64();
            const bool ok = mbar_wait_lean(turn == 0 ? done : never, 0u, flag_addr, 70 + turn);
            if (lane == 0) { result[turn] = ok; cycles[turn] = clock64() - t0; }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) result[3] = flag;
}

extern "C" int run_waits(int* result, long long* cycles, void* stream) {
    wait_kernel<<<1, 96, 0, (cudaStream_t)stream>>>(result, cycles);
    return (int)cudaGetLastError();
}
