// Matrix product of the true 32-bit path: out[m, n] = sum_k x[m, k] * w[n, k] (+ bias[n]) (+ residual[m, n]), all float, for matrices of fewer
// than 1024 features or columns (larger ones: linear_f32_tc.cu, unless a caller names a kernel of this file).
//
// The order of every sum is fixed by K alone, so that a row of the result has the same bits in every batch, whichever
// kernel below computes it: K is cut into blocks of 32; within a block the even and the odd k are two fused
// multiply-add chains in ascending k (the two halves of a packed fma.rn.f32x2), the block's sum is even + odd, and the
// blocks' sums are added in ascending order. Elements past K count as zeros. (Shorter chains than one over all of K:
// the error against 64 bits is smaller, at K = 8960 by about three times.)
//
// Up to 8 rows, `gemv32_kernel`: bound by reading w. A CTA takes 16 (or 8) features; a thread owns one block of 32 of
// one feature in every 256 elements of K and multiplies it with all rows of x, so w is read from HBM once, by coalesced
// 16-byte asynchronous copies through a ring of stages, and nothing but the blocks' sums crosses threads. The copies'
// 16-byte units are placed in an XOR pattern so that eight threads reading eight blocks side by side meet eight banks.
// Where the caller says that no kernel still running writes w (a loaded weight), the ring's first weights are requested before
// the kernel waits for its predecessor.
//
// (17920 x 1536: 1 row 20 us = 5.5 TB/s, 3 rows 31, 8 rows 44, bound by the reads of x from shared memory; 1536 x 8960: 17, 25, 35.
// A single token's step of the 1.5B sizes on tiles of 64 x 64 with scalar reads and no copies in flight took 55.6 ms, its products now 2.)
//
// More rows, `tile32_kernel`: bound by the FMA units, which run at 57 % (512 rows, 17920 x 1536: 670 us = 42 TFLOP/s; scalar FMAs
// in the same order 730; the products of a 512-token step of the 1.5B sizes 37 ms, on the tiles before 88). Operands stay K-contiguous in shared memory (rows padded to 36
// floats: eight rows read side by side meet eight banks); a 16-byte read feeds two packed FMAs without any shuffling
// of halves, which is why a block's chains are even and odd k. Tiles of 64 x 64 (8 x 4 results a thread), or smaller ones
// where those would leave SMs idle.
#include "common.cuh"

IB_DEFINE_LAST_ERROR()

namespace {

constexpr int BLOCK_K = 32;               // elements of K whose sum is formed before it is added to the total

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }
// 16 (or 4) bytes into shared memory, zeros where !ok (nothing is read then).
__device__ __forceinline__ void copy16(uint32_t dst, const float* src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copy4(uint32_t dst, const float* src, bool ok) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(ok ? 4 : 0) : "memory");
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void wait_groups() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// One 16-byte unit (4 elements of K from k on) of a row, at `dst`. VEC: K and the base are multiples of 16 bytes.
template <bool VEC>
__device__ __forceinline__ void copy_unit(uint32_t dst, const float* base, const float* row, int64_t k, int64_t K, bool live) {
    if constexpr (VEC) {
        const bool ok = live && k < K;
        copy16(dst, ok ? row + k : base, ok);
    } else {
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const bool ok = live && k + e < K;
            copy4(dst + 4u * e, ok ? row + k + e : base, ok);
        }
    }
}

using pair = unsigned long long;          // two floats: even k in the low half, odd k in the high one
__device__ __forceinline__ void fma2(pair& acc, pair a, pair b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float sum2(pair v) {
    return __uint_as_float(uint32_t(v)) + __uint_as_float(uint32_t(v >> 32));
}
__device__ __forceinline__ void lds_pairs(pair& a, pair& b, const float* at) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(at);
    a = v.x; b = v.y;
}

__device__ __forceinline__ void store_result(float v, int64_t m, int64_t n, int64_t N, const float* bias, const float* residual, float* out) {
    if (bias) v += bias[n];
    if (residual) v += residual[m * N + n];
    out[m * N + n] = v;
}

// ------------------------------------------------------------------------------------------------ up to 8 rows
constexpr int GK = 256, GBLOCKS = GK / BLOCK_K, GSTAGES = 4;   // K per stage, blocks of it, stages

template <int ROWS, int MT>
constexpr int gemv_smem() { return GSTAGES * (ROWS + MT) * GK * 4; }

template <int ROWS, int MT, bool VEC>
__global__ void __launch_bounds__(ROWS * GBLOCKS)
gemv32_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias, const float* residual,
              float* out, int M, int64_t N, int64_t K, int w_ready) {
    extern __shared__ __align__(128) float stages[];           // [GSTAGES][ROWS rows of w, MT rows of x][GK]
    constexpr int THREADS = ROWS * GBLOCKS, UNITS = GK / 4;
    __shared__ float sums[THREADS / 32][4][GBLOCKS][MT + 1];   // per warp: 4 features x 8 blocks x rows
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int blk = lane & 7, feature = tid >> 3;              // a warp: 4 features x 8 blocks
    const int64_t n0 = int64_t(blockIdx.x) * ROWS;
    const int steps = int((K + GK - 1) / GK);
    const uint32_t base = smem_u32(stages);
    constexpr uint32_t STAGE_BYTES = (ROWS + MT) * GK * 4;
    // unit u (16 bytes) of a row lies at its block's place ^ the block's number
    auto unit_place = [](int u) { return uint32_t((u & ~7) | ((u ^ (u >> 3)) & 7)) * 16u; };
    auto load_w = [&](int step) {
        const uint32_t dst = base + uint32_t(step % GSTAGES) * STAGE_BYTES;
#pragma unroll
        for (int i = 0; i < ROWS * UNITS / THREADS; i++) {
            const int u = tid + i * THREADS, r = u / UNITS, c = u % UNITS;
            copy_unit<VEC>(dst + uint32_t(r) * GK * 4u + unit_place(c), w, w + (n0 + r) * K, int64_t(step) * GK + 4 * c, K, n0 + r < N);
        }
    };
    auto load_x = [&](int step) {
        const uint32_t dst = base + uint32_t(step % GSTAGES) * STAGE_BYTES + ROWS * GK * 4u;
        for (int u = tid; u < MT * UNITS; u += THREADS) {
            const int r = u / UNITS, c = u % UNITS;
            copy_unit<VEC>(dst + uint32_t(r) * GK * 4u + unit_place(c), x, x + r * K, int64_t(step) * GK + 4 * c, K, r < M);
        }
    };
    if (!w_ready) ib::pdl_wait();
    for (int s = 0; s < GSTAGES - 1 && s < steps; s++) load_w(s);
    ib::pdl_wait();
    for (int s = 0; s < GSTAGES - 1; s++) {
        if (s < steps) load_x(s);
        commit();
    }
    ib::pdl_launch_dependents();
    float total = 0.0f;                                        // of row `blk` (where blk < MT)
    for (int step = 0; step < steps; step++) {
        wait_groups<GSTAGES - 2>();
        __syncthreads();                                       // the stage is there, and the one before it has been read
        if (step + GSTAGES - 1 < steps) { load_w(step + GSTAGES - 1); load_x(step + GSTAGES - 1); }
        commit();
        const float* stage = stages + (step % GSTAGES) * (ROWS + MT) * GK;
        const float *wrow = stage + feature * GK + blk * BLOCK_K, *xrow = stage + ROWS * GK + blk * BLOCK_K;
        pair acc[MT];
#pragma unroll
        for (int m = 0; m < MT; m++) acc[m] = 0;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            pair w0, w1;
            lds_pairs(w0, w1, wrow + (j ^ blk) * 4);
#pragma unroll
            for (int m = 0; m < MT; m++) {
                pair x0, x1;
                lds_pairs(x0, x1, xrow + m * GK + (j ^ blk) * 4);
                fma2(acc[m], w0, x0);
                fma2(acc[m], w1, x1);
            }
        }
        // the blocks' sums change hands: lane `blk` of a feature adds row blk's eight, ascending
        __syncwarp();
#pragma unroll
        for (int m = 0; m < MT; m++) sums[warp][lane >> 3][blk][m] = sum2(acc[m]);
        __syncwarp();
        if (blk < MT) {
#pragma unroll
            for (int b = 0; b < GBLOCKS; b++) total += sums[warp][lane >> 3][b][blk];
        }
    }
    wait_groups<0>();
    const int64_t n = n0 + feature;
    if (blk < MT && blk < M && n < N) store_result(total, blk, n, N, bias, residual, out);
}

// ------------------------------------------------------------------------------------------------ more rows
constexpr int TSTAGES = 3, PITCH = BLOCK_K + 4;                // floats between rows of a stage

template <int TM, int TN>
constexpr int tile_smem() { return TSTAGES * (8 * TM + 16 * TN) * PITCH * 4; }

// 128 threads, warps 2 x 2, a warp's threads 4 x 8, a thread TM x TN results: a tile of 8 TM x 16 TN.
template <int TM, int TN, bool VEC>
__global__ void __launch_bounds__(128, TM * TN > 16 ? 3 : 4)
tile32_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias, const float* residual,
              float* out, int64_t M, int64_t N, int64_t K) {
    extern __shared__ __align__(128) float stages[];           // [TSTAGES][BM rows of x, BN rows of w][PITCH]
    constexpr int BM = 8 * TM, BN = 16 * TN, UNITS = BLOCK_K / 4;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t m0 = int64_t(blockIdx.y) * BM, n0 = int64_t(blockIdx.x) * BN;
    const int steps = int((K + BLOCK_K - 1) / BLOCK_K);
    const uint32_t base = smem_u32(stages);
    constexpr uint32_t STAGE_BYTES = (BM + BN) * PITCH * 4, ROW = PITCH * 4;
    auto load = [&](int step) {
        const uint32_t dst = base + uint32_t(step % TSTAGES) * STAGE_BYTES;
#pragma unroll
        for (int i = 0; i < (BM + BN) * UNITS / 128; i++) {
            const int u = tid + i * 128, r = u / UNITS, c = u % UNITS;
            const bool is_x = r < BM;                          // (the same for the whole warp)
            const int64_t row = is_x ? m0 + r : n0 + r - BM;
            copy_unit<VEC>(dst + uint32_t(r) * ROW + c * 16u, is_x ? x : w, (is_x ? x : w) + row * K, int64_t(step) * BLOCK_K + 4 * c, K,
                           row < (is_x ? M : N));
        }
    };
    ib::pdl_wait();
    for (int s = 0; s < TSTAGES - 1; s++) {
        if (s < steps) load(s);
        commit();
    }
    const int ty = (warp >> 1) * 4 * TM + (lane >> 3), tx = (warp & 1) * 8 * TN + (lane & 7);      // rows ty + 4 i, columns tx + 8 j
    float total[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) total[i][j] = 0.0f;
    for (int step = 0; step < steps; step++) {
        wait_groups<TSTAGES - 2>();
        __syncthreads();
        if (step + TSTAGES - 1 < steps) load(step + TSTAGES - 1);
        commit();
        const float *xs = stages + ((step % TSTAGES) * (BM + BN) + ty) * PITCH, *ws = stages + ((step % TSTAGES) * (BM + BN) + BM + tx) * PITCH;
        pair acc[TM][TN];
#pragma unroll
        for (int i = 0; i < TM; i++)
#pragma unroll
            for (int j = 0; j < TN; j++) acc[i][j] = 0;
#pragma unroll
        for (int c = 0; c < UNITS; c++) {
            pair b0[TN], b1[TN];
#pragma unroll
            for (int j = 0; j < TN; j++) lds_pairs(b0[j], b1[j], ws + 8 * j * PITCH + 4 * c);
#pragma unroll
            for (int i = 0; i < TM; i++) {
                pair a0, a1;
                lds_pairs(a0, a1, xs + 4 * i * PITCH + 4 * c);
#pragma unroll
                for (int j = 0; j < TN; j++) { fma2(acc[i][j], b0[j], a0); fma2(acc[i][j], b1[j], a1); }
            }
        }
#pragma unroll
        for (int i = 0; i < TM; i++)
#pragma unroll
            for (int j = 0; j < TN; j++) total[i][j] += sum2(acc[i][j]);
    }
    wait_groups<0>();
    ib::pdl_launch_dependents();
#pragma unroll
    for (int i = 0; i < TM; i++) {
        const int64_t m = m0 + ty + 4 * i;
#pragma unroll
        for (int j = 0; j < TN; j++) {
            const int64_t n = n0 + tx + 8 * j;
            if (m < M && n < N) store_result(total[i][j], m, n, N, bias, residual, out);
        }
    }
}

struct Args {
    const float *x, *w, *bias, *residual;
    float* out;
    int64_t M, N, K;
    int w_ready;
};

template <int ROWS, int MT, bool VEC>
int launch_gemv(const Args& a, cudaStream_t stream) {
    static ib::PerDevice allowed;
    if (const int rc = ib::allow_smem(allowed, "linear_f32", gemv32_kernel<ROWS, MT, VEC>, gemv_smem<ROWS, MT>())) return rc;
    return ib::launch("linear_f32", gemv32_kernel<ROWS, MT, VEC>, dim3(unsigned((a.N + ROWS - 1) / ROWS)), dim3(ROWS * GBLOCKS),
                      size_t(gemv_smem<ROWS, MT>()), stream, 1u, a.x, a.w, a.bias, a.residual, a.out, int(a.M), a.N, a.K, a.w_ready);
}

template <int ROWS, bool VEC>
int launch_gemv_rows(const Args& a, cudaStream_t stream) {
    if (a.M == 1) return launch_gemv<ROWS, 1, VEC>(a, stream);
    if (a.M == 2) return launch_gemv<ROWS, 2, VEC>(a, stream);
    if (a.M <= 4) return launch_gemv<ROWS, 4, VEC>(a, stream);
    return launch_gemv<ROWS, 8, VEC>(a, stream);
}

template <int TM, int TN, bool VEC>
int launch_tile(const Args& a, cudaStream_t stream) {
    static ib::PerDevice allowed;
    if (const int rc = ib::allow_smem(allowed, "linear_f32", tile32_kernel<TM, TN, VEC>, tile_smem<TM, TN>())) return rc;
    const dim3 grid{unsigned((a.N + 16 * TN - 1) / (16 * TN)), unsigned((a.M + 8 * TM - 1) / (8 * TM)), 1u};
    if (grid.y > 65535) return ib::fail(IB_ERR_ARG, "linear_f32: too many rows (%lld)", (long long)a.M);
    return ib::launch("linear_f32", tile32_kernel<TM, TN, VEC>, grid, dim3(128), size_t(tile_smem<TM, TN>()), stream, 1u, a.x, a.w, a.bias,
                      a.residual, a.out, a.M, a.N, a.K);
}

template <bool VEC>
int dispatch(const Args& a, int kind, int sms, cudaStream_t stream) {
    if (kind == 0) {
        if (a.M <= 8) {
            // 16 features a CTA share a row of x among twice as many threads; 8 where those CTAs leave SMs idle (N = 1536, K = 8960:
            // 8 rows 34.5 against 36.4 us, one row 17.3 to 17.7 either way; with 3 rows 25.4 either way, N = 2048, K = 1536: 5.0 and 5.1).
            // Of the sizes that come here, with 16 and with 8 features: 896 x 896 one row 2.5 and 2.7, 3 rows 3.4 and 3.3, 8 rows 4.7 and 4.2;
            // 896 x 4864 9.1 and 9.2, 13.5 and 12.5, 19.6 and 16.7; 9728 x 896 8.5 and 8.6, 14.2 and 13.6, 19.4 and 17.4
            kind = (a.N + 15) / 16 >= 2LL * sms || (a.M > 1 && a.M <= 4) ? 1 : 2;
        } else {
            // The larger a thread's share the fewer shared-memory reads per FMA, but a CTA alone on its SM is bound by its own
            // chain (1.07 us per 32 elements of K with 8 x 4 results a thread, 0.66 with 4 x 4, 0.43 with 4 x 2): 64 x 64 and
            // 32 x 64 need about one and a half CTAs an SM (512 rows, N = 1536: 192 and 384 tiles, 94 and 77 us; 256 rows: 192
            // tiles of 32 x 64 take 54 us, 384 of 32 x 32 48), and 64-row tiles win by 8 % where they pad no more rows
            // (N = 17920: 87 rows 175 against 147 us, 128 rows 177 against 194). Of the sizes that come here, 64 x 64, 32 x 64 and 32 x 32:
            // 896 x 4864 9 rows 158, 98 and 64 us, 512 rows 165, 166 and 193, 2,048 rows 552, 530 and 595; 9728 x 896 64 rows 57, 47 and 46,
            // 128 rows 80, 74 and 79, 2,048 rows 805, 895 and 1,103: the choice is within 9 % of the best
            const int64_t big = ((a.M + 63) / 64) * ((a.N + 63) / 64), mid = ((a.M + 31) / 32) * ((a.N + 63) / 64);
            const bool pads = (a.M + 63) / 64 * 64 * 100 > (a.M + 31) / 32 * 32 * 108;
            kind = big * 5 >= 8LL * sms && !pads ? 3 : (mid * 2 >= 3LL * sms ? 4 : 5);
        }
    }
    if ((kind == 1 || kind == 2) && a.M > 8) return ib::fail(IB_ERR_ARG, "linear_f32: this kernel takes up to 8 rows");
    switch (kind) {
        case 1: return launch_gemv_rows<16, VEC>(a, stream);
        case 2: return launch_gemv_rows<8, VEC>(a, stream);
        case 3: return launch_tile<8, 4, VEC>(a, stream);
        case 4: return launch_tile<4, 4, VEC>(a, stream);
        case 5: return launch_tile<4, 2, VEC>(a, stream);
    }
    return ib::fail(IB_ERR_ARG, "linear_f32: unknown kernel %d", kind);
}

}  // namespace

// kind: 0 = chosen from the sizes; 1, 2 = up to 8 rows with 16 / 8 features a CTA; 3, 4, 5 = tiles of 64 x 64, 32 x 64, 32 x 32.
// Every kind gives the same bits. residual may be out. w_ready: 1 = no kernel that may still run writes w (it may be read before
// this kernel's predecessor has ended), 0 = w may come from the predecessor.
IB_EXPORT int ib_linear_f32(const float* x, const float* w, const float* bias, const float* residual, float* out, int64_t M, int64_t N,
                            int64_t K, int kind, int sm_count, int w_ready, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return IB_OK;
    if (K <= 0) return ib::fail(IB_ERR_ARG, "linear_f32: K must be positive");
    const int64_t lim = 1LL << 31;                             // of the blocks of 32 elements of K, and of CTAs with 8 features each
    if (N >= 8 * lim || K >= BLOCK_K * lim) return ib::fail(IB_ERR_ARG, "linear_f32: more features or columns than the kernels count");
    const Args a{x, w, bias, residual, out, M, N, K, w_ready};
    const int sms = sm_count > 0 ? sm_count : 148;
    const bool vec = K % 4 == 0 && ((uintptr_t(x) | uintptr_t(w)) & 15) == 0;
    return vec ? dispatch<true>(a, kind, sms, stream) : dispatch<false>(a, kind, sms, stream);
}
