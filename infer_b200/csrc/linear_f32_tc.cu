// Matrix product of the true 32-bit path on the 5th-generation tensor cores:
// out[m, n] = sum_k x[m, k] * w[n, k] (+ bias[n]) (+ residual[m, n]), all float, for matrices of at least 1024 x 1024.
//
// Every float is cut into three bfloat16 numbers, v = v1 + v2 2^-8 + v3 2^-16 (each the rounding of what the ones before it
// leave; three times eight bits hold a float's 24), on its way from global to shared memory, and a product becomes six of
// the tensor cores': w1 x1 in one accumulator, w1 x2 + w2 x1 in a second (weight 2^-8) and w1 x3 + w2 x2 + w3 x1 in a third
// (2^-16). What is left out is w2 x3 + w3 x2 (and w3 x3, below 2^-33): |v2| 2^-8 is at most 2^-8 of v and |v3| 2^-16 at most 2^-17 (both
// where v is just above a power of two), hence below 2^-24 of a product, for random operands mostly below 2^-26. The powers of two keep the
// small parts out of the subnormal range. A result that is not finite (an operand that is not, or too large a sum or part) is computed again
// by plain multiply-adds, so that infinities and NaN come out as they do there.
//
// The tensor core's additions do not round as a float addition does, so few of them follow one another where it counts: the
// first accumulator starts anew every 64 elements of K and is added to a float in registers; the other two, whose errors
// weigh 2^-8, run over a group of such blocks. Groups (at most 8, from N, K and the device's SMs) are added in ascending order. A result
// does not depend on how many rows x has, nor on which CTA forms which group: on one device a row's bits are the same in every batch.
// Error against 64 bits (norm over norm), multiply-adds in brackets: normal operands 0.94e-7 (1.3e-7) at K = 1024, 1.2e-7 (3.1e-7) at 8960.
// The tensor core truncates, so operands of one sign have errors of one sign, -0.7e-7 on average (1e-10), in norm 0.92e-7 (0.90e-7) at
// K = 1024 and 0.95e-7 (2.6e-7) at 8960; scales e^(3 normal) apart -3.3e-7 (-0.1e-7), 2.0e-7 (0.7e-7) and 1.7e-7 (5.9e-7); normal w and
// widely scaled x 1.4e-7 (1.2e-7) and 1.2e-7 (4.0e-7). Closer than multiply-adds from K = 3584 on, whatever the operands; below, on those
// that a model has.
// us on multiply-adds -> here: 512 rows, 17920 x 1536 669 -> 267, 1536 x 8960 440 -> 165; 16 rows 54 -> 28 and 117 -> 21; 3 rows 30 -> 27
// and 24 -> 21. One and two rows lose: 18.7 -> 27.4, 16.8 -> 20.9, 2048 x 1536 4.3 -> 9.1, 4608 x 3584 11.9 -> 29.9, 151936 x 1536 129 -> 230.
// (A row's bits must not depend on the batch, so they come here too: what prompts gain is 2 to 6 times that.) The line at 1024 x 1024: below
// it the tiles leave most SMs idle.
//
// A CTA (544 threads, one an SM) forms 128 features x NT tokens (features on the tensor memory's 128 lanes). Sixteen warps load a
// block of 64 elements of K into registers a block or two ahead, cut and store it as six swizzled operand tiles, and add up the
// accumulator of the block before, while the seventeenth warp issues the block's 16 MMAs. The sixteen warps' instructions bound
// it as much as anything: pairs of floats go through packed arithmetic, and addresses advance by addition. A few rows (NT = 16) are bound by
// the chain of a worker's round (cut, fence, arrive, see that the MMAs of the block before are done, add: 1,770 cycles, also where w came through
// a ring of asynchronous copies and where a tile had half the features: 17920 x 1536 at one row 32 us that way), 64 rows and more by the workers' instructions beside shared
// memory's bandwidth (per block 72 KB stored and 112 KB read by the MMAs against 768 cycles of the tensor pipe).
// Where the tiles are fewer than the SMs, the groups of a tile go to the CTAs of a cluster: each pushes its groups' sums to
// the CTAs that own their columns, through distributed shared memory, and after one cluster barrier the owners add them.
#include "common.cuh"
#include "tc_ops.cuh"

IB_DEFINE_LAST_ERROR()

namespace {

using namespace ib::tc;

constexpr int BM = 128, BK = 64;                 // features of a tile, elements of K in a block
constexpr int WARPS = 16, WORKERS = WARPS * 32, THREADS = WORKERS + 32;
constexpr int MAX_GROUPS = 8;
constexpr int A_BYTES = BM * BK * 2;
constexpr int SMEM_MOST = 226 * 1024;
constexpr int STATUS_TIMEOUT = 131;

template <int NT> struct Cfg {
    static constexpr int B_BYTES = NT * BK * 2;
    static constexpr int STAGE_BYTES = 3 * A_BYTES + 3 * B_BYTES;
    static constexpr int TMEM_COLS = NT >= 64 ? 512 : (NT >= 32 ? 256 : 128);    // six accumulators of NT columns
    static constexpr int COLS = NT / 4;          // columns of a warp
    static constexpr int A_UNITS = BM * BK / 4 / WORKERS;                        // 16-byte units of w a thread and block
    static constexpr int B_UNITS = (NT * BK / 4 + WORKERS - 1) / WORKERS;        // ... of x (NT = 16: half of the threads)
    static constexpr int DEPTH = NT >= 64 ? 1 : 2;                               // blocks requested ahead
};

template <int N> __device__ __forceinline__ void tmem_ld(uint32_t taddr, float* v);
template <> __device__ __forceinline__ void tmem_ld<4>(uint32_t taddr, float* v) {
    uint32_t r[4];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 4; j++) v[j] = __uint_as_float(r[j]);
}
template <> __device__ __forceinline__ void tmem_ld<8>(uint32_t taddr, float* v) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 8; j++) v[j] = __uint_as_float(r[j]);
}
template <> __device__ __forceinline__ void tmem_ld<16>(uint32_t taddr, float* v) {
    uint32_t r[16];
    tmem_ld16(taddr, r);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 16; j++) v[j] = __uint_as_float(r[j]);
}

// Four elements of a row, the first of them at `at`. VEC: 16-byte aligned. ONCE: w, which is read once a step.
template <bool VEC, bool ONCE>
__device__ __forceinline__ float4 load_unit(const float* at) {
    float4 v;
    if constexpr (VEC) {
        if constexpr (ONCE) asm volatile("ld.global.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(at));
        else asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(at));
    } else {
        v.x = at[0]; v.y = at[1]; v.z = at[2]; v.w = at[3];
    }
    return v;
}
// The same where only `n` of the four (or none) are in the row: zeros for the others.
__device__ __forceinline__ float4 load_some(const float* at, int n) {
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (n > 0) v.x = at[0];
    if (n > 1) v.y = at[1];
    if (n > 2) v.z = at[2];
    if (n > 3) v.w = at[3];
    return v;
}

// Two floats rounded to bfloat16: the first in the low half.
__device__ __forceinline__ uint32_t round2(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}
// Two floats side by side in 64 bits, for the packed forms of the arithmetic.
using pair = unsigned long long;
__device__ __forceinline__ pair pack(uint32_t lo, uint32_t hi) { return (pair(hi) << 32) | lo; }
// (v - h) 256, exactly: h is v rounded to bfloat16 (two of them in 32 bits).
__device__ __forceinline__ void rest(float& a, float& b, uint32_t h) {
    constexpr pair MINUS = 0xbf800000bf800000ull, SCALE = 0x4380000043800000ull;
    pair v = pack(__float_as_uint(a), __float_as_uint(b));
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(v) : "l"(pack(h << 16, h & 0xffff0000u)), "l"(MINUS));
    asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(v) : "l"(SCALE));
    a = __uint_as_float(uint32_t(v));
    b = __uint_as_float(uint32_t(v >> 32));
}

// The three parts of four elements, eight bytes each, `part` bytes apart.
__device__ __forceinline__ void store_parts(uint8_t* at, uint32_t part, float4 v) {
    uint2 p;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        p.x = round2(v.x, v.y);
        p.y = round2(v.z, v.w);
        *reinterpret_cast<uint2*>(at + i * part) = p;
        if (i < 2) { rest(v.x, v.y, p.x); rest(v.z, v.w, p.y); }
    }
}

struct Params {
    const float *x, *w, *bias, *residual;
    float* out;
    int64_t M, N, K;
    int blocks, groups, per_cta;                 // blocks of K, groups of them, groups a CTA forms
    int share;                                   // CTAs of a tile (a cluster)
    int* status;
    int w_ready;
};

__device__ __forceinline__ uint32_t map_cluster(uint32_t local_smem, uint32_t rank) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local_smem), "r"(rank));
    return remote;
}

// One result by plain multiply-adds, in the order of linear_f32.cu: blocks of 32 elements of K, even and odd k apart, then the blocks' sums
// in ascending order. A warp takes 16 blocks at a time through its shared memory (two lanes a block, blocks 34 floats apart: no two lanes
// meet in a bank). Every lane has the result.
constexpr int PLAIN_BLOCKS = 16, PLAIN_PITCH = 34, PLAIN_FLOATS = 2 * PLAIN_BLOCKS * PLAIN_PITCH;
__device__ __forceinline__ float plain_product(const float* x, const float* w, int64_t K, float* mem, int lane) {
    float total = 0.0f;
    float* mem_x = mem + PLAIN_BLOCKS * PLAIN_PITCH;
    for (int64_t k0 = 0; k0 < K; k0 += PLAIN_BLOCKS * 32) {
        __syncwarp();                                         // the blocks before have been read
#pragma unroll
        for (int b = 0; b < PLAIN_BLOCKS; b++) {
            const int64_t k = k0 + b * 32 + lane;
            mem[b * PLAIN_PITCH + lane] = k < K ? w[k] : 0.0f;
            mem_x[b * PLAIN_PITCH + lane] = k < K ? x[k] : 0.0f;
        }
        __syncwarp();
        const int at = (lane >> 1) * PLAIN_PITCH + (lane & 1);
        float sum = 0.0f;
#pragma unroll
        for (int j = 0; j < 32; j += 2) sum = fmaf(mem[at + j], mem_x[at + j], sum);
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        if (__any_sync(0xffffffffu, isnan(sum))) return __int_as_float(0x7fffffff);
#pragma unroll
        for (int b = 0; b < PLAIN_BLOCKS; b++) total += __shfl_sync(0xffffffffu, sum, 2 * b);
    }
    return total;
}

// Whether a row holds a NaN (asked by a whole warp).
__device__ __forceinline__ bool has_nan(const float* row, int64_t K, int lane) {
    bool found = false;
#pragma unroll 8
    for (int64_t k = lane; k < K; k += 32) found |= isnan(row[k]);
    return __any_sync(0xffffffffu, found) != 0;
}

static_assert(WARPS * PLAIN_FLOATS * 4 <= 2 * Cfg<16>::STAGE_BYTES, "the warps' blocks lie in the operand stages");

template <int NT, bool VEC>
__global__ void __launch_bounds__(THREADS, 1)
linear32_tc_kernel(const Params p) {
    using C = Cfg<NT>;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bars[4];    // full[2], done[2]
    __shared__ uint32_t slot, failed, again;
    uint8_t* stages = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    // [own column][128 features] the groups' sum so far, or, where a tile is shared, [group][own column][128 features] each group's
    float* recv = reinterpret_cast<float*>(stages + 2 * C::STAGE_BYTES);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, int(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int rank = blockIdx.x;                              // in the cluster
    // (the last tile of features is a whole one too: what it shares with the one before, it does not store)
    const int64_t n_first = int64_t(blockIdx.y) * BM, n0 = min(n_first, p.N - BM), m0 = int64_t(blockIdx.z) * NT;
    const int g_begin = rank * p.per_cta, g_end = g_begin + p.per_cta;
    auto first_block = [&](int g) { return int(int64_t(g) * p.blocks / p.groups); };
    const int b0 = first_block(g_begin), nb = first_block(g_end) - b0;
    const uint32_t bar0 = smem_u32(bars);
    auto full = [&](int b) { return bar0 + 8u * (b & 1); };
    auto done = [&](int b) { return bar0 + 16u + 8u * (b & 1); };

    if (tid == 0) {
        for (int i = 0; i < 2; i++) { mbar_init(full(i), WARPS); mbar_init(done(i), 1); }
        failed = again = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == WARPS) {
        tmem_alloc(smem_u32(&slot), C::TMEM_COLS);
        tmem_relinquish();
    }

    // Unit `unit` of rows row0, row0 + 32, ... of either operand; the pointers advance with the blocks. (In place of rows past x's
    // last one others are read: what they lead to is not stored.)
    const int unit = tid & 15, row0 = (tid >> 4) & 31;
    constexpr int ROW_STEP = WORKERS / 16;
    const bool worker = warp < WARPS, has_x = worker && (NT * 16 >= WORKERS || tid < NT * 16);
    float4 wq[C::DEPTH][C::A_UNITS], xq[C::DEPTH][C::B_UNITS];
    const int64_t k_first = int64_t(b0) * BK + unit * 4, step = ROW_STEP * p.K;
    const float* pw = p.w + (n0 + row0) * p.K + k_first;
    const float* px = p.x + min(m0 + row0, p.M - 1) * p.K + k_first;
    const int64_t x_step = m0 + row0 + ROW_STEP < p.M ? step : 0;
    const int whole = int(min(int64_t(nb), p.K / BK - b0));   // blocks that lie inside K
    const int tail = int(p.K - p.K / BK * BK) - unit * 4;     // elements of this unit in the block that does not
    auto load_w = [&](int b, int d) {
        const float* at = pw;
        if (b < whole) {
#pragma unroll
            for (int i = 0; i < C::A_UNITS; i++, at += step) wq[d][i] = load_unit<VEC, true>(at);
        } else {
#pragma unroll
            for (int i = 0; i < C::A_UNITS; i++, at += step) wq[d][i] = load_some(at, tail);
        }
        pw += BK;
    };
    auto load_x = [&](int b, int d) {
        if (has_x) {
            const float* at = px;
            if (b < whole) {
#pragma unroll
                for (int i = 0; i < C::B_UNITS; i++, at += x_step) xq[d][i] = load_unit<VEC, false>(at);
            } else {
#pragma unroll
                for (int i = 0; i < C::B_UNITS; i++, at += x_step) xq[d][i] = load_some(at, tail);
            }
        }
        px += BK;
    };
    if (!p.w_ready) ib::pdl_wait();
    if (worker) {
#pragma unroll
        for (int d = 0; d < C::DEPTH; d++)
            if (d < nb) load_w(d, d);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // (the CTAs of a cluster push into one another's shared memory: each has to have started)
    if (p.share > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    const uint32_t tmem = slot;
    ib::pdl_wait();
    if (worker) {
#pragma unroll
        for (int d = 0; d < C::DEPTH; d++)
            if (d < nb) load_x(d, d);
    }
    if (p.share > 1) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");

    const uint32_t lanes = tmem + (uint32_t((warp & 3) * 32) << 16) + uint32_t(warp >> 2) * C::COLS;
    const int row = (warp & 3) * 32 + lane, col0 = (warp >> 2) * C::COLS;              // this thread's feature and first token
    const int own_cols = NT / p.share;                        // columns that a CTA of the cluster adds and stores
    float acc[C::COLS];
#pragma unroll
    for (int j = 0; j < C::COLS; j++) acc[j] = 0.0f;
    int g = g_begin, g_last = first_block(g_begin + 1) - b0;  // the group at hand; the first block of the next one
    bool ok = true;
    if (warp == WARPS) {
        // ------------------------------------------------------------------------------------------------ MMA issuer
        constexpr uint32_t one = make_idesc(NT, false), two = make_idesc(2 * NT, false);
        const bool leader = elect_one();
        bool fresh = true;                                    // the next block's MMAs are their group's first
        for (int b = 0; b < nb; b++) {
            if (b == g_last) { g++; g_last = first_block(g + 1) - b0; fresh = true; }
            if (!mbar_wait_each(full(b), uint32_t(b >> 1) & 1u)) { ok = false; break; }
            tc_fence_after();
            const uint32_t a = smem_u32(stages) + uint32_t(b & 1) * C::STAGE_BYTES, x = a + 3 * A_BYTES;
            const uint32_t c0 = tmem + uint32_t(b & 1) * NT, c12 = tmem + uint32_t(2 + 2 * ((g - g_begin) & 1)) * NT;
            const uint64_t w1 = make_desc(a, 16, 1024), w2 = make_desc(a + A_BYTES, 16, 1024), w3 = make_desc(a + 2 * A_BYTES, 16, 1024);
            const uint64_t x1 = make_desc(x, 16, 1024), x2 = make_desc(x + C::B_BYTES, 16, 1024);
            if (leader) {
#pragma unroll
                for (int k = 0; k < BK / 16; k++) {
                    const uint64_t o = uint64_t(2 * k);       // 16 elements = 32 bytes = 2 units of the address field
                    umma_f16(c0, w1 + o, x1 + o, one, k > 0);
                    umma_f16(c12, w1 + o, x2 + o, two, (!fresh || k > 0) ? 1u : 0u);
                    umma_f16(c12, w2 + o, x1 + o, two, 1u);
                    umma_f16(c12 + NT, w3 + o, x1 + o, one, 1u);
                }
                umma_commit(done(b));
            }
            __syncwarp();
            fresh = false;
        }
    } else {
        // ------------------------------------------------------------------------------------------------ workers
        const uint32_t place = uint32_t(row0) * 128u + ((uint32_t(unit >> 1) ^ uint32_t(row0 & 7)) << 4) + uint32_t(unit & 1) * 8u;   // (32 rows on: the same pattern)
        // adds what block b left in its accumulator; at the end of a group also the two of the group
        auto add_up = [&](int b) {
            if (!mbar_wait_warp(done(b), uint32_t(b >> 1) & 1u)) { ok = false; return; }
            tc_fence_after();
            float v[C::COLS];
            tmem_ld<C::COLS>(lanes + uint32_t(b & 1) * NT, v);
#pragma unroll
            for (int j = 0; j < C::COLS; j++) acc[j] += v[j];
            if (b + 1 == g_last) {
                float u[C::COLS];
                const uint32_t c12 = lanes + uint32_t(2 + 2 * ((g - g_begin) & 1)) * NT;
                tmem_ld<C::COLS>(c12, v);
                tmem_ld<C::COLS>(c12 + NT, u);
                int owner = col0 / own_cols, own = col0 - owner * own_cols;
#pragma unroll
                for (int j = 0; j < C::COLS; j++) {
                    const float sum = acc[j] + fmaf(u[j], 1.0f / 65536.0f, v[j] * (1.0f / 256.0f));
                    if (p.share > 1) {
                        const uint32_t at = map_cluster(smem_u32(recv) + uint32_t((g * own_cols + own) * BM + row) * 4u, uint32_t(owner));
                        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(at), "f"(sum) : "memory");
                        if (++own == own_cols) { own = 0; owner++; }
                    } else {
                        float* at = recv + (col0 + j) * BM + row;
                        *at = g > 0 ? *at + sum : sum;
                    }
                    acc[j] = 0.0f;
                }
                g++;
                g_last = first_block(g + 1) - b0;
            }
            tc_fence_before();
        };
        auto next_block = [&](int b, int d) {
            // (the stage is free: its last MMAs, block b - 2's, were waited for when that block was added up)
            uint8_t* at = stages + (b & 1) * C::STAGE_BYTES + place;
            if (b + C::DEPTH < whole) {
                // a unit's registers take the next load as soon as it is stored: that load has the whole of a block's time
                const float *from = pw, *from_x = px;
#pragma unroll
                for (int i = 0; i < C::A_UNITS; i++, from += step) {
                    store_parts(at + i * (ROW_STEP * 128), A_BYTES, wq[d][i]);
                    wq[d][i] = load_unit<VEC, true>(from);
                }
                if (has_x) {
#pragma unroll
                    for (int i = 0; i < C::B_UNITS; i++, from_x += x_step) {
                        store_parts(at + 3 * A_BYTES + i * (ROW_STEP * 128), C::B_BYTES, xq[d][i]);
                        xq[d][i] = load_unit<VEC, false>(from_x);
                    }
                }
                pw += BK;
                px += BK;
            } else {
#pragma unroll
                for (int i = 0; i < C::A_UNITS; i++) store_parts(at + i * (ROW_STEP * 128), A_BYTES, wq[d][i]);
                if (has_x) {
#pragma unroll
                    for (int i = 0; i < C::B_UNITS; i++) store_parts(at + 3 * A_BYTES + i * (ROW_STEP * 128), C::B_BYTES, xq[d][i]);
                }
                if (b + C::DEPTH < nb) { load_w(b + C::DEPTH, d); load_x(b + C::DEPTH, d); }
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(full(b));
            if (b > 0) add_up(b - 1);
        };
        for (int b = 0; b < nb && ok; b += C::DEPTH) {
#pragma unroll
            for (int d = 0; d < C::DEPTH; d++)
                if (b + d < nb && ok) next_block(b + d, d);
        }
        ib::pdl_launch_dependents();
        if (ok) add_up(nb - 1);
    }
    if (!ok && lane == 0) { atomicExch(p.status, STATUS_TIMEOUT); *reinterpret_cast<volatile uint32_t*>(&failed) = 1; }

    // Feature tid & 127 of own columns tid / 128, + 4, ..., four columns at a time; what is added to the first four's sums is requested
    // before the barrier.
    const int64_t n = n0 + (tid & (BM - 1));
    const bool storing = worker && n >= n_first;
    const float bias = storing && p.bias ? p.bias[n] : 0.0f;
    const int slots = p.share > 1 ? p.groups : 1;
    float res[4];
    auto request = [&](int c0) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int c = c0 + (tid >> 7) + 4 * i;
            const int64_t m = m0 + rank * own_cols + c;
            res[i] = storing && p.residual && c < own_cols && m < p.M ? p.residual[m * p.N + n] : 0.0f;
        }
    };
    request(0);
    __syncwarp();
    if (p.share > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    else __syncthreads();
    if (storing && !*reinterpret_cast<volatile uint32_t*>(&failed)) {
        for (int c0 = 0; c0 < own_cols; c0 += 16) {
            if (c0) request(c0);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int c = c0 + (tid >> 7) + 4 * i;
                const int64_t m = m0 + rank * own_cols + c;
                if (c < own_cols && m < p.M) {
                    float v = 0.0f;
                    for (int h = 0; h < slots; h++) v += recv[(h * own_cols + c) * BM + (tid & (BM - 1))];
                    if (!isfinite(v)) {
                        *reinterpret_cast<volatile uint32_t*>(&again) = 1;
                        continue;
                    }
                    if (p.bias) v += bias;
                    if (p.residual) v += res[i];
                    p.out[m * p.N + n] = v;
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == WARPS) {
        tc_fence_after();
        tmem_dealloc(tmem, C::TMEM_COLS);
    } else if (*reinterpret_cast<volatile uint32_t*>(&again)) {
        // Results that are not finite, by multiply-adds: a warp takes 8 of the 128 features of every column, so that a column whose
        // token holds a NaN or an infinity is spread over all warps; where it holds a NaN, all of the column's results are known at once.
        // (One row that holds a NaN or an infinity, calls by themselves: 17920 x 1536, 1, 16 and 512 rows 45 and 69, 46 and 68, 292 and 320 us,
        // all finite 44, 43, 285; 1536 x 8960, 16 rows 43 and 192 against 34. A thread for each of them took 204, 204, 456 and 827.)
        const int f = warp * (BM / WARPS) + (lane & 7);
        const int64_t nf = n0 + f;
        float* mem = reinterpret_cast<float*>(stages) + warp * PLAIN_FLOATS;           // (every MMA that read the stages has been waited for)
        for (int c0 = 0; c0 < own_cols; c0 += 4) {
            const int c = c0 + (lane >> 3);
            const int64_t m = m0 + rank * own_cols + c;
            float v = 0.0f;
            if (c < own_cols && m < p.M && nf >= n_first)
                for (int h = 0; h < slots; h++) v += recv[(h * own_cols + c) * BM + f];
            const bool mine = !isfinite(v);
            const uint32_t todo = __ballot_sync(0xffffffffu, mine);
            for (int q = 0; q < 4; q++) {
                uint32_t here = (todo >> (8 * q)) & 0xffu;
                const float* row = p.x + (m0 + rank * own_cols + c0 + q) * p.K;
                if ((here & (here - 1)) && has_nan(row, p.K, lane)) {
                    if (mine && (lane >> 3) == q) v = __int_as_float(0x7fffffff);
                    continue;
                }
                for (; here; here &= here - 1) {
                    const int j = __ffs(here) - 1;
                    const float total = plain_product(row, p.w + (n0 + warp * (BM / WARPS) + j) * p.K, p.K, mem, lane);
                    if (lane == 8 * q + j) v = total;
                }
            }
            if (mine) {
                if (p.bias) v += p.bias[nf];
                if (p.residual) v += p.residual[m * p.N + nf];
                p.out[m * p.N + nf] = v;
            }
        }
    }
}

struct Plan { int nt, groups, share; };

// Groups: as many as give the tiles of features alone work for every SM, a power of two, at most 8, of at least two blocks each. From N, K
// and the device alone, never from M: the order of a row's sums must not depend on how many rows there are.
int group_count(int64_t N, int64_t blocks, int sms) {
    const int64_t tiles = (N + BM - 1) / BM;
    int g = 1;
    while (g < MAX_GROUPS && tiles * g * 2 <= sms && blocks >= 4 * g) g *= 2;
    return g;
}

int smem_bytes(int nt, int groups, int share) {
    const int recv = nt * BM * 4 * (share > 1 ? groups : 1) / share;
    return 2 * 3 * (A_BYTES + nt * BK * 2) + 1024 + recv;
}

Plan make_plan(int64_t M, int64_t N, int64_t K, int sms) {
    Plan q;
    const int64_t blocks = (K + BK - 1) / BK;
    q.groups = group_count(N, blocks, sms);
    q.nt = M <= 16 ? 16 : (M <= 32 ? 32 : 64);
    const int64_t tiles = ((N + BM - 1) / BM) * ((M + q.nt - 1) / q.nt);
    // How many CTAs share a tile: the number whose rounds over the SMs take least, a CTA's start and end counted as four blocks
    // and the cluster's meeting as two more. (A CTA of a cluster holds every group's sums of its columns.)
    q.share = 1;
    int64_t best = 0;
    for (int z = 1; z <= q.groups; z *= 2) {
        if (smem_bytes(q.nt, q.groups, z) > SMEM_MOST) continue;
        // (of the SMs, clusters of four and eight cannot use a seventh)
        const int64_t at_once = z == 1 ? sms : (z == 2 ? sms - 4 : (sms - sms / 7) / z * z);
        const int64_t rounds = (tiles * z + at_once - 1) / at_once;
        const int64_t cost = rounds * ((blocks + z - 1) / z + 4 + (z > 1 ? 2 : 0));
        if (best == 0 || cost < best) { best = cost; q.share = z; }
    }
    return q;
}

template <int NT, bool VEC>
int launch_tc(const Params& p, const Plan& q, cudaStream_t stream) {
    static ib::PerDevice allowed;
    if (const int rc = ib::allow_smem(allowed, "linear_f32_tc", linear32_tc_kernel<NT, VEC>, SMEM_MOST)) return rc;
    const int64_t rows = (p.M + NT - 1) / NT, cols = (p.N + BM - 1) / BM;
    if (rows > 65535 || cols > 65535) return ib::fail(IB_ERR_ARG, "linear_f32_tc: %lld x %lld results are too many", (long long)p.M, (long long)p.N);
    return ib::launch("linear_f32_tc", linear32_tc_kernel<NT, VEC>, dim3(unsigned(q.share), unsigned(cols), unsigned(rows)), dim3(THREADS),
                      size_t(smem_bytes(NT, q.groups, q.share)), stream, unsigned(q.share), p);
}

template <bool VEC>
int launch_nt(const Params& p, const Plan& q, cudaStream_t stream) {
    if (q.nt == 16) return launch_tc<16, VEC>(p, q, stream);
    if (q.nt == 32) return launch_tc<32, VEC>(p, q, stream);
    return launch_tc<64, VEC>(p, q, stream);
}

}  // namespace

// 1 where this kernel takes the matrix: a matter of N and K alone, so that every batch of rows takes the same way.
IB_EXPORT int ib_linear_f32_tc_takes(int64_t N, int64_t K) {
    return N >= 1024 && K >= 1024 && N <= 65535LL * BM && K < (1LL << 31) ? 1 : 0;
}

// residual may be out. w_ready: as in ib_linear_f32.
IB_EXPORT int ib_linear_f32_tc(const float* x, const float* w, const float* bias, const float* residual, float* out, int64_t M, int64_t N,
                               int64_t K, int sm_count, int w_ready, int* status, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return IB_OK;
    if (!ib_linear_f32_tc_takes(N, K)) return ib::fail(IB_ERR_ARG, "linear_f32_tc: a matrix of %lld x %lld is not taken", (long long)N, (long long)K);
    if (!status) return ib::fail(IB_ERR_ARG, "linear_f32_tc: a status word is required");
    const Plan q = make_plan(M, N, K, sm_count > 0 ? sm_count : 148);
    const Params p{x, w, bias, residual, out, M, N, K, int((K + BK - 1) / BK), q.groups, q.groups / q.share, q.share, status, w_ready};
    const bool vec = K % 4 == 0 && ((uintptr_t(x) | uintptr_t(w)) & 15) == 0;
    return vec ? launch_nt<true>(p, q, stream) : launch_nt<false>(p, q, stream);
}
