// Matrix product of the true 32-bit path on the 5th-generation tensor cores:
// out[m, n] = sum_k x[m, k] * w[n, k] (+ bias[n]) (+ residual[m, n]), all float, for matrices of at least 1024 x 1024.
//
// Every float is cut into three bfloat16 numbers, v = v1 + v2 2^-8 + v3 2^-16 (each the rounding of what the ones before it
// leave; three times eight bits hold a float's 24), on its way from global to shared memory, and a product becomes six of
// the tensor cores': w1 x1 in one accumulator, w1 x2 + w2 x1 in a second (weight 2^-8) and w1 x3 + w2 x2 + w3 x1 in a third
// (2^-16). What is left out (w2 x3, w3 x2, w3 x3) is below 2^-26 of a product. The powers of two keep the small parts out of
// the subnormal range. A result that is not finite (an operand that is not, or too large a sum or part) is computed again by
// plain multiply-adds, so that infinities and NaN come out as they do there.
//
// The tensor core's additions do not round as a float addition does, so few of them follow one another where it counts: the
// first accumulator starts anew every 64 elements of K and is added to a float in registers; the other two, whose errors
// weigh 2^-8, run over a group of such blocks. Groups (at most 8, from N and K alone) are added in ascending order. A result
// does not depend on how many rows x has, nor on which CTA forms which group: a row's bits are the same in every batch.
//
// A CTA (512 threads, one an SM) forms 128 features x NT tokens (features on the tensor memory's 128 lanes). Its warps load a
// block of 64 elements of K into registers two blocks ahead, cut and store it as six swizzled operand tiles, the first warp
// issues the block's 16 MMAs, and meanwhile all add up the accumulator of the block before. A few rows (NT = 16) are bound by
// the reads of w; 64 rows and more by shared memory's bandwidth (per block 72 KB stored and 112 KB read by the MMAs
// against 768 cycles of the tensor pipe).
// Where the tiles are fewer than the SMs, the groups of a tile go to the CTAs of a cluster: each pushes its groups' sums to
// the CTAs that own their columns, through distributed shared memory, and after one cluster barrier the owners add them.
#include "common.cuh"
#include "tc_ops.cuh"

IB_DEFINE_LAST_ERROR()

namespace {

using namespace ib::tc;

constexpr int BM = 128, BK = 64;                 // features of a tile, elements of K in a block
constexpr int WARPS = 16, THREADS = WARPS * 32;
constexpr int MAX_GROUPS = 8;
constexpr int A_BYTES = BM * BK * 2;
constexpr int SMEM_MOST = 226 * 1024;
constexpr int STATUS_TIMEOUT = 131;
constexpr int DEPTH = 2;                         // blocks requested ahead

template <int NT> struct Cfg {
    static constexpr int B_BYTES = NT * BK * 2;
    static constexpr int STAGE_BYTES = 3 * A_BYTES + 3 * B_BYTES;
    static constexpr int TMEM_COLS = NT >= 64 ? 512 : (NT >= 32 ? 256 : 128);    // six accumulators of NT columns
    static constexpr int COLS = NT / 4;          // columns of a warp
    static constexpr int A_UNITS = BM * BK / 4 / THREADS;                        // 16-byte units of w a thread and block
    static constexpr int B_UNITS = (NT * BK / 4 + THREADS - 1) / THREADS;        // ... of x (NT = 16: half of the threads)
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

// Four elements of a row from k on; past its end others of the row, which `cleared` takes out (a load without a condition is in
// flight until its value is used). VEC: 16-byte aligned, K a multiple of 4. ONCE: w, which is read once a step.
template <bool VEC, bool ONCE>
__device__ __forceinline__ float4 load_unit(const float* row, int64_t k, int64_t K) {
    float4 v;
    if constexpr (VEC) {
        const float* at = row + (k < K ? k : K - 4);
        if constexpr (ONCE) asm volatile("ld.global.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(at));
        else v = *reinterpret_cast<const float4*>(at);
    } else {
        v.x = row[k < K ? k : K - 1]; v.y = row[k + 1 < K ? k + 1 : K - 1];
        v.z = row[k + 2 < K ? k + 2 : K - 1]; v.w = row[k + 3 < K ? k + 3 : K - 1];
    }
    return v;
}
__device__ __forceinline__ float4 cleared(float4 v, int64_t k, int64_t K) {
    if (k >= K) v.x = 0.0f;
    if (k + 1 >= K) v.y = 0.0f;
    if (k + 2 >= K) v.z = 0.0f;
    if (k + 3 >= K) v.w = 0.0f;
    return v;
}

// Two floats rounded to bfloat16: the first in the low half.
__device__ __forceinline__ uint32_t round2(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float low_half(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float high_half(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

// The three parts of four elements, eight bytes each, `part` bytes apart.
__device__ __forceinline__ void store_parts(uint8_t* at, uint32_t part, float4 v) {
    uint2 p;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        p.x = round2(v.x, v.y);
        p.y = round2(v.z, v.w);
        *reinterpret_cast<uint2*>(at + i * part) = p;
        if (i < 2) {
            v.x = (v.x - low_half(p.x)) * 256.0f; v.y = (v.y - high_half(p.x)) * 256.0f;
            v.z = (v.z - low_half(p.y)) * 256.0f; v.w = (v.w - high_half(p.y)) * 256.0f;
        }
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

// One result by plain multiply-adds.
__device__ __noinline__ float plain_product(const float* x, const float* w, int64_t K) {
    float total = 0.0f;
    for (int64_t k0 = 0; k0 < K; k0 += 32) {
        float block = 0.0f;
        for (int64_t k = k0; k < K && k < k0 + 32; k++) block = fmaf(x[k], w[k], block);
        total += block;
    }
    return total;
}

template <int NT, bool VEC>
__global__ void __launch_bounds__(THREADS, 1)
linear32_tc_kernel(const Params p) {
    using C = Cfg<NT>;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bars[4];    // full[2], done[2]
    __shared__ uint32_t slot, failed;
    uint8_t* stages = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* recv = stages + 2 * C::STAGE_BYTES;              // [group][own column][128 features] where a tile is shared
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, int(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int rank = blockIdx.x;                              // in the cluster
    const int64_t n0 = int64_t(blockIdx.y) * BM, m0 = int64_t(blockIdx.z) * NT;
    const int g_begin = rank * p.per_cta, g_end = g_begin + p.per_cta;
    auto first_block = [&](int g) { return int(int64_t(g) * p.blocks / p.groups); };
    const int b0 = first_block(g_begin), nb = first_block(g_end) - b0;
    const uint32_t bar0 = smem_u32(bars);
    auto full = [&](int b) { return bar0 + 8u * (b & 1); };
    auto done = [&](int b) { return bar0 + 16u + 8u * (b & 1); };

    if (tid == 0) {
        for (int i = 0; i < 2; i++) { mbar_init(full(i), WARPS); mbar_init(done(i), 1); }
        failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        tmem_alloc(smem_u32(&slot), C::TMEM_COLS);
        tmem_relinquish();
    }

    const int unit = tid & 15, row0 = tid >> 4;               // unit u of rows row0, row0 + 32, ...
    constexpr int ROW_STEP = THREADS / 16;
    const bool has_x = NT * 16 >= THREADS || tid < NT * 16;
    float4 wq[DEPTH][C::A_UNITS], xq[DEPTH][C::B_UNITS];
    // (rows past the last one are read from it: what they lead to is not stored)
    auto load_w = [&](int b, int d) {
        const int64_t k = int64_t(b0 + b) * BK + unit * 4;
#pragma unroll
        for (int i = 0; i < C::A_UNITS; i++) wq[d][i] = load_unit<VEC, true>(p.w + min(n0 + row0 + i * ROW_STEP, p.N - 1) * p.K, k, p.K);
    };
    auto load_x = [&](int b, int d) {
        const int64_t k = int64_t(b0 + b) * BK + unit * 4;
        if (has_x) {
#pragma unroll
            for (int i = 0; i < C::B_UNITS; i++) xq[d][i] = load_unit<VEC, false>(p.x + min(m0 + row0 + i * ROW_STEP, p.M - 1) * p.K, k, p.K);
        }
    };
    if (!p.w_ready) ib::pdl_wait();
#pragma unroll
    for (int d = 0; d < DEPTH; d++)
        if (d < nb) load_w(d, d);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // (the CTAs of a cluster push into one another's shared memory: each has to have started)
    if (p.share > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    const uint32_t tmem = slot;
    ib::pdl_wait();
#pragma unroll
    for (int d = 0; d < DEPTH; d++)
        if (d < nb) load_x(d, d);
    if (p.share > 1) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");

    const bool leader = elect_one();
    const uint32_t lanes = tmem + (uint32_t((warp & 3) * 32) << 16) + uint32_t(warp >> 2) * C::COLS;
    const int row = (warp & 3) * 32 + lane, col0 = (warp >> 2) * C::COLS;              // this thread's feature and first token
    const int own_cols = NT / p.share;                        // columns that a CTA of the cluster adds and stores
    float acc[C::COLS], total[C::COLS];
#pragma unroll
    for (int j = 0; j < C::COLS; j++) acc[j] = total[j] = 0.0f;
    int g = g_begin, g_last = first_block(g_begin + 1) - b0;  // the group that is being added up; the first block of the next one
    int mma_g = g_begin, mma_last = g_last;                   // the same for the MMAs, which are a block ahead
    bool fresh = true;                                        // the next block's MMAs are their group's first
    bool ok = true;
    // the first warp: block b's MMAs, once every warp has stored its part of the operands
    auto multiply = [&](int b) {
        constexpr uint32_t one = make_idesc(NT, false), two = make_idesc(2 * NT, false);
        if (b == mma_last) { mma_g++; mma_last = first_block(mma_g + 1) - b0; fresh = true; }
        if (!mbar_wait_each(full(b), uint32_t(b >> 1) & 1u)) { ok = false; return; }
        tc_fence_after();
        const uint32_t a = smem_u32(stages) + uint32_t(b & 1) * C::STAGE_BYTES, x = a + 3 * A_BYTES;
        const uint32_t c0 = tmem + uint32_t(b & 1) * NT, c12 = tmem + uint32_t(2 + 2 * ((mma_g - g_begin) & 1)) * NT;
        const uint64_t w1 = make_desc(a, 16, 1024), w2 = make_desc(a + A_BYTES, 16, 1024), w3 = make_desc(a + 2 * A_BYTES, 16, 1024);
        const uint64_t x1 = make_desc(x, 16, 1024), x2 = make_desc(x + C::B_BYTES, 16, 1024);
        if (leader) {
#pragma unroll
            for (int k = 0; k < BK / 16; k++) {
                const uint64_t o = uint64_t(2 * k);           // 16 elements = 32 bytes = 2 units of the address field
                umma_f16(c0, w1 + o, x1 + o, one, k > 0);
                umma_f16(c12, w1 + o, x2 + o, two, (!fresh || k > 0) ? 1u : 0u);
                umma_f16(c12, w2 + o, x1 + o, two, 1u);
                umma_f16(c12 + NT, w3 + o, x1 + o, one, 1u);
            }
            umma_commit(done(b));
        }
        __syncwarp();
        fresh = false;
    };
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
                    total[j] += sum;
                }
                acc[j] = 0.0f;
            }
            g++;
            g_last = first_block(g + 1) - b0;
        }
        tc_fence_before();
    };
    auto step = [&](int b, int d) {
        // (the stage is free: its last MMAs, block b - 2's, were waited for when that block was added up)
        uint8_t* stage = stages + (b & 1) * C::STAGE_BYTES;
        auto place = [&](int r) { return uint32_t(r) * 128u + ((uint32_t(unit >> 1) ^ uint32_t(r & 7)) << 4) + uint32_t(unit & 1) * 8u; };
        const int64_t k = int64_t(b0 + b) * BK + unit * 4;
        if (int64_t(b0 + b + 1) * BK > p.K) {
#pragma unroll
            for (int i = 0; i < C::A_UNITS; i++) wq[d][i] = cleared(wq[d][i], k, p.K);
#pragma unroll
            for (int i = 0; i < C::B_UNITS; i++) xq[d][i] = cleared(xq[d][i], k, p.K);
        }
#pragma unroll
        for (int i = 0; i < C::A_UNITS; i++) store_parts(stage + place(row0 + i * ROW_STEP), A_BYTES, wq[d][i]);
        if (has_x) {
#pragma unroll
            for (int i = 0; i < C::B_UNITS; i++) store_parts(stage + 3 * A_BYTES + place(row0 + i * ROW_STEP), C::B_BYTES, xq[d][i]);
        }
        fence_proxy_async();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(full(b));
        if (b + DEPTH < nb) { load_w(b + DEPTH, d); load_x(b + DEPTH, d); }
        if (warp == 0) multiply(b);
        if (b > 0 && ok) add_up(b - 1);
    };
    for (int b = 0; b < nb && ok; b += DEPTH) {
#pragma unroll
        for (int d = 0; d < DEPTH; d++)
            if (b + d < nb && ok) step(b + d, d);
    }
    ib::pdl_launch_dependents();
    if (ok) add_up(nb - 1);
    if (!ok && lane == 0) { atomicExch(p.status, STATUS_TIMEOUT); *reinterpret_cast<volatile uint32_t*>(&failed) = 1; }

    auto finish = [&](float v, int64_t m, int64_t n, float bias, float res) {
        if (!isfinite(v)) v = plain_product(p.x + m * p.K, p.w + n * p.K, p.K);
        if (p.bias) v += bias;
        if (p.residual) v += res;
        p.out[m * p.N + n] = v;
    };
    if (p.share > 1) {
        // feature tid & 127 of own columns tid / 128, + 4, ...; what is added to the sums is requested before the barrier
        constexpr int MOST = 4;                               // (a CTA owns at most 16 columns)
        const int64_t n = n0 + (tid & (BM - 1));
        const bool n_ok = n < p.N;
        const float bias = p.bias && n_ok ? p.bias[n] : 0.0f;
        float res[MOST];
#pragma unroll
        for (int i = 0; i < MOST; i++) {
            const int c = (tid >> 7) + 4 * i;
            const int64_t m = m0 + rank * own_cols + c;
            res[i] = p.residual && n_ok && c < own_cols && m < p.M ? p.residual[m * p.N + n] : 0.0f;
        }
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (n_ok && !*reinterpret_cast<volatile uint32_t*>(&failed)) {
            const float* sums = reinterpret_cast<const float*>(recv);
#pragma unroll
            for (int i = 0; i < MOST; i++) {
                const int c = (tid >> 7) + 4 * i;
                const int64_t m = m0 + rank * own_cols + c;
                if (c < own_cols && m < p.M) {
                    float v = 0.0f;
                    for (int h = 0; h < p.groups; h++) v += sums[(h * own_cols + c) * BM + (tid & (BM - 1))];
                    finish(v, m, n, bias, res[i]);
                }
            }
        }
    } else {
        const int64_t n = n0 + row;
        if (n < p.N && !*reinterpret_cast<volatile uint32_t*>(&failed)) {
            const float bias = p.bias ? p.bias[n] : 0.0f;
            float res[C::COLS];
#pragma unroll
            for (int j = 0; j < C::COLS; j++) {
                const int64_t m = m0 + col0 + j;
                res[j] = p.residual && m < p.M ? p.residual[m * p.N + n] : 0.0f;
            }
#pragma unroll
            for (int j = 0; j < C::COLS; j++) {
                const int64_t m = m0 + col0 + j;
                if (m < p.M) finish(total[j], m, n, bias, res[j]);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, C::TMEM_COLS);
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
    const int recv = share > 1 ? nt * BM * 4 * groups / share : 0;
    return 2 * 3 * (A_BYTES + nt * BK * 2) + 1024 + recv;
}

Plan make_plan(int64_t M, int64_t N, int64_t K, int sms) {
    Plan q;
    const int64_t blocks = (K + BK - 1) / BK;
    q.groups = group_count(N, blocks, sms);
    q.nt = M <= 16 ? 16 : (M <= 32 ? 32 : 64);
    const int64_t tiles = ((N + BM - 1) / BM) * ((M + q.nt - 1) / q.nt);
    // How many CTAs share a tile: the number whose rounds over the SMs take least, a CTA's start and end counted as four blocks
    // and the cluster's meeting as two more. (A CTA stores at most 16 columns, and holds every group's sums of those.)
    q.share = 1;
    int64_t best = 0;
    for (int z = 1; z <= q.groups; z *= 2) {
        if (z > 1 && (q.nt / z > 16 || smem_bytes(q.nt, q.groups, z) > SMEM_MOST)) continue;
        const int64_t rounds = (tiles * z + sms - 1) / sms;
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
