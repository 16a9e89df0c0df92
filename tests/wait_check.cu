// The warp's waits of tc_ops.cuh by themselves (test_waits_gpu.py): a barrier that nobody arrives on, and one that completes when some
// lanes have given up and others have not. Every wait here is bounded: at most 32 x 8 tries, or 2^16 of about a microsecond.
#include "tc_ops.cuh"

using namespace ib::tc;

// out: per case 32 lanes: 1 = the wait was told a success, 0 = it ran out; for the last case what the other warp had stored before.
__global__ void __launch_bounds__(64) wait_check_kernel(int* out) {
    __shared__ __align__(8) unsigned long long bars[3];
    __shared__ volatile int data;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 3; i++) mbar_init(smem_u32(&bars[i]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        data = 0;
    }
    __syncthreads();
    if (warp == 0) {
        // nobody arrives on the first barrier; every lane has another limit
        out[0 * 32 + lane] = mbar_wait_each(smem_u32(&bars[0]), 0, 1u + 8u * lane);
        out[1 * 32 + lane] = mbar_wait_warp(smem_u32(&bars[0]), 0, 8);
    }
    __syncthreads();
    if (warp == 0) {
        // the second completes after about 100 us: half of the lanes have given up by then
        out[2 * 32 + lane] = mbar_wait_each(smem_u32(&bars[1]), 0, lane < 16 ? 1u : 1u << 16);
        // it has completed
        out[3 * 32 + lane] = mbar_wait_each(smem_u32(&bars[1]), 0, 1u << 16);
    } else {
        for (int i = 0; i < 100; i++) __nanosleep(1000);
        if (lane == 0) mbar_arrive(smem_u32(&bars[1]));
    }
    __syncthreads();
    if (warp == 0) {
        const int ok = mbar_wait_warp(smem_u32(&bars[2]), 0, 1u << 16);
        out[4 * 32 + lane] = ok ? data : -1;
    } else {
        for (int i = 0; i < 20; i++) __nanosleep(1000);
        if (lane == 0) {
            data = 7;
            mbar_arrive(smem_u32(&bars[2]));
        }
    }
}

extern "C" __attribute__((visibility("default"))) int wait_check(int* out, cudaStream_t stream) {
    wait_check_kernel<<<1, 64, 0, stream>>>(out);
    return int(cudaGetLastError());
}
