// fp32 products of many rows on the tensor cores: C (M,N) = act(A (M,K) W (N,K)^T + bias), both operands cut into bf16 parts.
//
// A 24-bit significand is three bf16 numbers: x1 = bf16(x), x2 = bf16(x - x1), x3 = x - x1 - x2, exactly (G. Henry, P. T. P. Tang,
// A. Heinecke, Leveraging the bfloat16 artificial intelligence datatype for higher-precision computations, ARITH 2019).  Of the nine
// products of parts the six down to 2^-18 of the largest are taken; the three left out are below 2^-26 of |a b|, less than the
// rounding of a partial sum of an fp32 chain.  A weight that is a bf16 number (a bf16 checkpoint run in fp32) has one part, and
// three products are all there are.  (Exactly from 2^-109 on: below that x3, from 2^-117 on x2 as well, falls out of bf16's range,
// and what is lost stays below 2^-134.)
//
// bn_linear_f32 cuts both operands anew in every call, so that a weight may be written to at any time, and by anything, between
// two calls; which tiles of the weight have one part and which three is found out on the way.  Cutting a weight of 2048 x 7424 takes
// 21 us with three parts and 12 us with one.
//
// The tensor cores add into fp32 accumulators with truncation, which over a long K would cost more than a chain of FMAs does.
// So an accumulator takes 64 k only, the small products first and x1 w1 last, and these sums are added up in registers, rounded
// to nearest: 4 truncations at full size in an accumulator, K / 64 roundings in a sum, where a chain has K.
//
// A row with a sum that is not finite (an infinity or a NaN among the operands, a part that overflows bf16, a sum that does) is
// worked out again, 32 columns at a time, as chains of FMAs from the fp32 operands (300 x 7424 -> 1032, 0.13 ms: with an infinity
// in two of the rows 0.67 ms, in all of them 3.7 ms, with NaN in half of them 0.14 ms).
//
// CTA = one tile of 128 x BN at a time, persistent: warps 0-7 add accumulators up and store (a thread: one row, half of the
// columns), warp 8 issues MMAs, warp 9 loads tiles of 64 k by TMA; two accumulators.
#include <float.h>
#include <limits.h>

#include "common.cuh"
#include "hybrid.cuh"
#include "ptx.cuh"
#include "tcgen05.cuh"
#include "tma.cuh"

namespace bn {

using namespace ptx;

constexpr int MS_BM = 128, MS_BK = 64, MS_THREADS = 320, MS_PARTS = 3;

template <int BN> struct SplitShape {
    static constexpr int A_BYTES = MS_BM * MS_BK * 2, B_BYTES = BN * MS_BK * 2;
    static constexpr int STAGE_BYTES = MS_PARTS * (A_BYTES + B_BYTES);
    static constexpr int NSTAGE = 204800 / STAGE_BYTES;
    static constexpr int SMEM_BYTES = 1024 + NSTAGE * STAGE_BYTES;
    static constexpr uint32_t TMEM_COLS = 2 * BN;
};

struct SplitParams {
    const float *a, *w, *bias;
    float* c;
    int* error_word;
    const uint8_t* counts;         // how many parts the weight has, 1 or 3, in every tile of BN rows x 64 k; null: w_parts everywhere
    int64_t a_ld, w_ld;
    int M, N, K, act, w_parts;
    bool aligned;                  // a's and w's rows start on 16-byte boundaries
};

// The rows m0 + i of the set bits i of `rows`, as chains: a warp, a lane per column (n the lane's), four rows at a time and 8 k of
// every operand in flight.  A chain that has become a NaN stays one, so rows that are all NaN end at once.  Nobody waits for it
// for long: at worst (every row of a tile, no NaN) about 0.5 us per k, where the CTA's other warps give up after 2 s.
__device__ __noinline__ void redo_rows(const SplitParams& p, uint32_t rows, int m0, int n) {
    constexpr int ROWS = 4, AHEAD = 2;           // K is a multiple of 8
    const bool in = n < p.N;
    const float* w = p.w + (in ? n : 0) * p.w_ld;
    auto load = [&](const float* from, float (&v)[4]) {
        if (p.aligned) load4(from, v);
        else
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = from[e];
    };
    while (rows) {
        int m[ROWS];
        const float* a[ROWS];
        float sum[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {                       // (a row again where none is left)
            m[r] = rows ? m0 + __ffs(rows) - 1 : m[0];
            rows &= rows - 1;
            a[r] = p.a + m[r] * p.a_ld;
            sum[r] = 0.f;
        }
        for (int k0 = 0; k0 < p.K; k0 += 4 * AHEAD) {
            float y[AHEAD][4], x[ROWS][AHEAD][4];
#pragma unroll
            for (int j = 0; j < AHEAD; ++j) {
                load(w + k0 + 4 * j, y[j]);
#pragma unroll
                for (int r = 0; r < ROWS; ++r) load(a[r] + k0 + 4 * j, x[r][j]);
            }
#pragma unroll
            for (int j = 0; j < AHEAD; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e)
#pragma unroll
                    for (int r = 0; r < ROWS; ++r) sum[r] = fmaf(x[r][j][e], y[j][e], sum[r]);
            bool done = true;
#pragma unroll
            for (int r = 0; r < ROWS; ++r) done &= sum[r] != sum[r];
            if (__all_sync(0xffffffffu, done || !in)) break;
        }
        if (in)
#pragma unroll
            for (int r = 0; r < ROWS; ++r) p.c[(size_t)m[r] * p.N + n] = activation_exact(p.act, p.bias ? sum[r] + p.bias[n] : sum[r]);
    }
}

template <int BN>
__global__ void __launch_bounds__(MS_THREADS, 1)
mm_split_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_w,
                const __grid_constant__ SplitParams p) {
    using Sh = SplitShape<BN>;
    constexpr int NSTAGE = Sh::NSTAGE;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bar_full[NSTAGE], bar_empty[NSTAGE], bar_acc_full[2], bar_acc_empty[2];
    __shared__ uint32_t s_tmem_base;
    __shared__ int s_abort;

    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int tiles_m = (p.M + MS_BM - 1) / MS_BM, tiles_n = (p.N + BN - 1) / BN, n_tiles = tiles_m * tiles_n;
    const int k_steps = (p.K + MS_BK - 1) / MS_BK;
    auto w_parts = [&](int tile_n, int ks) { return p.counts ? (int)p.counts[(size_t)tile_n * k_steps + ks] : p.w_parts; };

    if (tid == 0) {
        for (int s = 0; s < NSTAGE; ++s) {
            mbar_init(smem_u32(&bar_full[s]), 1);
            mbar_init(smem_u32(&bar_empty[s]), 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(smem_u32(&bar_acc_full[i]), 1);
            mbar_init(smem_u32(&bar_acc_empty[i]), 8);
        }
        s_abort = 0;
        fence_mbar_init();
    }
    if (warp == 8) {
        tc::tmem_alloc(smem_u32(&s_tmem_base), Sh::TMEM_COLS);
        tc::tmem_relinquish();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = s_tmem_base;
    grid_dependency_wait();                                    // a programmatic dependent, as the cut in front of it

    if (warp == 9) {
        if (lane == 0) {
            prefetch_tensormap(&tmap_a);
            prefetch_tensormap(&tmap_w);
            uint32_t it = 0;
            bool ok = true;
            for (int t = blockIdx.x; ok && t < n_tiles; t += gridDim.x) {
                const int m0 = t % tiles_m * MS_BM, n0 = t / tiles_m * BN;
                for (int ks = 0; ks < k_steps; ++ks, ++it) {
                    const int stage = it % NSTAGE, parts = w_parts(t / tiles_m, ks);
                    ok = mbar_wait(smem_u32(&bar_empty[stage]), ((it / NSTAGE) & 1u) ^ 1u, &s_abort);
                    if (!ok) break;
                    const uint32_t full = smem_u32(&bar_full[stage]), sA = smem0 + stage * Sh::STAGE_BYTES, sW = sA + MS_PARTS * Sh::A_BYTES;
                    mbar_arrive_expect_tx(full, MS_PARTS * Sh::A_BYTES + parts * Sh::B_BYTES);
                    // part q of A is rows q M .. q M + M - 1 of its map: a tile's rows beyond M are rows that are not stored
#pragma unroll
                    for (int q = 0; q < MS_PARTS; ++q) tma_load_2d(sA + q * Sh::A_BYTES, &tmap_a, ks * MS_BK, q * p.M + m0, full);
                    for (int q = 0; q < parts; ++q) tma_load_2d(sW + q * Sh::B_BYTES, &tmap_w, ks * MS_BK, q * p.N + n0, full);
                }
            }
        }
    } else if (warp == 8) {
        constexpr uint32_t IDESC = tc::idesc_bf16(MS_BM, BN, 0);
        const uint64_t d0 = tc::smem_desc_sw128(0);
        uint32_t it = 0;
        bool ok = true;
        for (int t = blockIdx.x; ok && t < n_tiles; t += gridDim.x) {
            for (int ks = 0; ks < k_steps; ++ks, ++it) {
                const uint32_t acc = it & 1u, stage = it % NSTAGE;
                const int parts = w_parts(t / tiles_m, ks);
                ok = mbar_wait(smem_u32(&bar_acc_empty[acc]), ((it >> 1) & 1u) ^ 1u, &s_abort) &&
                     mbar_wait(smem_u32(&bar_full[stage]), (it / NSTAGE) & 1u, &s_abort);
                if (!ok) break;
                if (elect_one()) {
                    tc::fence_after_sync();
                    const uint32_t s0 = smem0 + stage * Sh::STAGE_BYTES;
                    // (part of A, part of W), the smallest products first
                    constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PW[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
                    for (int q = 0; q < 6; ++q) {
                        if (PW[q] >= parts) continue;
                        const uint32_t sA = s0 + PA[q] * Sh::A_BYTES, sW = s0 + MS_PARTS * Sh::A_BYTES + PW[q] * Sh::B_BYTES;
#pragma unroll
                        for (int kk = 0; kk < MS_BK / 16; ++kk)
                            tc::mma_ss(tmem + acc * BN, d0 + (uint64_t)((sA >> 4) + kk * 2), d0 + (uint64_t)((sW >> 4) + kk * 2), IDESC,
                                       q > 0 || kk > 0);
                    }
                    tc::commit(smem_u32(&bar_empty[stage]));
                    tc::commit(smem_u32(&bar_acc_full[acc]));
                }
                __syncwarp();
            }
        }
    } else {
        constexpr int COLS = BN / 2;                           // this thread's columns of its row
        const int row = warp % 4 * 32 + lane, col = warp / 4 * COLS;
        const uint32_t tbase = tmem + ((uint32_t)(warp % 4 * 32) << 16) + col;
        uint32_t local = 0;
        bool ok = true;
        for (int t = blockIdx.x; ok && t < n_tiles; t += gridDim.x) {
            const int gm = t % tiles_m * MS_BM + row, n0 = t / tiles_m * BN + col;
            uint64_t sum[COLS / 2];
#pragma unroll
            for (int i = 0; i < COLS / 2; ++i) sum[i] = 0;
            for (int ks = 0; ks < k_steps; ++ks, ++local) {
                const uint32_t acc = local & 1u;
                ok = mbar_wait(smem_u32(&bar_acc_full[acc]), (local >> 1) & 1u, &s_abort);
                if (!ok) break;
                tc::fence_after_sync();
#pragma unroll
                for (int c = 0; c < COLS / 32; ++c) {
                    uint32_t r[32];
                    tc::ld32(tbase + acc * BN + c * 32, r);
                    tc::wait_ld(r);
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        sum[c * 16 + i] = add_f32x2(sum[c * 16 + i], pack_f32x2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])));
                }
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&bar_acc_empty[acc]));
            }
            if (!ok) break;
            float* crow = p.c + (size_t)gm * p.N + n0;
            const bool late = p.act != BN_ACT_NONE && p.act != BN_ACT_RELU2;
            uint32_t rows[COLS / 32];                          // rows to work out again, for every 32 columns
#pragma unroll
            for (int c = 0; c < COLS / 32; ++c) {
                bool bad = false;
                if (gm < p.M) {
#pragma unroll
                    for (int k = c * 32; k < c * 32 + 32; k += 4)
                        if (n0 + k < p.N) {                    // N is a multiple of 8
                            float v[4], b[4] = {0.f, 0.f, 0.f, 0.f};
                            unpack_f32x2(sum[k / 2], v[0], v[1]);
                            unpack_f32x2(sum[k / 2 + 1], v[2], v[3]);
                            if (p.bias) load4(p.bias + n0 + k, b);
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                bad |= !(fabsf(v[e]) <= FLT_MAX);
                                v[e] += b[e];
                                if (p.act == BN_ACT_RELU2) v[e] = relu2(v[e]);
                            }
                            store4(crow + k, v);
                        }
                    if (late && !bad)
#pragma unroll 1
                        for (int k = c * 32; k < c * 32 + 32 && n0 + k < p.N; ++k) crow[k] = activation_exact(p.act, crow[k]);
                }
                rows[c] = __ballot_sync(0xffffffffu, bad);     // orders the stores above before those of redo_rows
            }
#pragma unroll
            for (int c = 0; c < COLS / 32; ++c)
                if (rows[c]) redo_rows(p, rows[c], gm - lane, n0 + c * 32 + lane);
            __syncwarp();
        }
    }

    tc::fence_before_sync();
    __syncthreads();
    if (tid == 0 && s_abort && p.error_word) atomicExch(p.error_word, BN_ERR_TIMEOUT);
    if (warp == 8) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem, Sh::TMEM_COLS);
    }
}

// the next part of 8 values, which become what it leaves of them; what is not finite in bf16 stays in the first part alone
__device__ __forceinline__ uint4 cut_part(float (&v)[8]) {
    uint32_t w[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        w[e] = pack_bf16(v[2 * e], v[2 * e + 1]);
        const float lo = bf16_lo(w[e]), hi = bf16_hi(w[e]);
        v[2 * e] = fabsf(lo) <= FLT_MAX ? v[2 * e] - lo : 0.f;
        v[2 * e + 1] = fabsf(hi) <= FLT_MAX ? v[2 * e + 1] - hi : 0.f;
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}
__device__ __forceinline__ void load8(const float* s, float (&v)[8]) {
    load4(s, *reinterpret_cast<float(*)[4]>(v));
    load4(s + 4, *reinterpret_cast<float(*)[4]>(v + 4));
}

// x (rows, cols) -> parts [3][rows][cols], cols a multiple of 8; `thread` of `threads`
__device__ __forceinline__ void cut_rows(const float* x, int64_t ld, __nv_bfloat16* parts, long long rows, int cols, long long thread,
                                         long long threads) {
    const long long n8 = rows * (cols / 8), plane = rows * cols;
    for (long long i = thread; i < n8; i += threads) {
        const long long r = i / (cols / 8);
        float v[8];
        load8(x + r * ld + (i - r * (cols / 8)) * 8, v);
#pragma unroll
        for (int q = 0; q < MS_PARTS; ++q) *reinterpret_cast<uint4*>(parts + q * plane + i * 8) = cut_part(v);
    }
}

__global__ void __launch_bounds__(256)
split_parts_kernel(const float* x, int64_t ld, __nv_bfloat16* parts, long long rows, int cols) {
    cut_rows(x, ld, parts, rows, cols, (long long)blockIdx.x * 256 + threadIdx.x, (long long)gridDim.x * 256);
}

// Both operands of a product.  A block has one tile of BN weight rows x 64 k in registers: where one part is all there is, the
// other two, which nobody will read, are not written.  The blocks behind those of the weight cut the rows of A.  The weight is
// read evict-first (cut and product of 64 rows, 7424 -> 2048 94 -> 80 us, 2048 -> 7424 38 -> 34).
struct CutParams {
    const float *a, *w;
    __nv_bfloat16 *a_parts, *w_parts;
    uint8_t* counts;
    int64_t a_ld, w_ld;
    int M, N, K, w_blocks;
};

template <int BN>
__global__ void __launch_bounds__(BN * 4)
cut_operands_kernel(const CutParams p) {
    grid_dependency_wait();
    grid_launch_dependents();
    if ((int)blockIdx.x >= p.w_blocks) {
        cut_rows(p.a, p.a_ld, p.a_parts, p.M, p.K, (long long)(blockIdx.x - p.w_blocks) * (BN * 4) + threadIdx.x,
                 (long long)(gridDim.x - p.w_blocks) * (BN * 4));
        return;
    }
    const int k_steps = (p.K + MS_BK - 1) / MS_BK, n0 = blockIdx.x / k_steps * BN + threadIdx.x / 8;
    const int k = blockIdx.x % k_steps * MS_BK + threadIdx.x % 8 * 8;
    float v[2][8];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int n = n0 + i * (BN / 2);
#pragma unroll
        for (int e = 0; e < 8; ++e) v[i][e] = 0.f;
        if (n < p.N && k < p.K) {                              // read once: the parts are what should stay in L2
            const float4* from = reinterpret_cast<const float4*>(p.w + n * p.w_ld + k);
            const float4 f0 = __ldcs(from), f1 = __ldcs(from + 1);
            v[i][0] = f0.x; v[i][1] = f0.y; v[i][2] = f0.z; v[i][3] = f0.w;
            v[i][4] = f1.x; v[i][5] = f1.y; v[i][6] = f1.z; v[i][7] = f1.w;
        }
    }
    auto store = [&](int part, int i, const uint4& x) {
        const int n = n0 + i * (BN / 2);
        if (n < p.N && k < p.K) *reinterpret_cast<uint4*>(p.w_parts + ((size_t)part * p.N + n) * p.K + k) = x;
    };
    bool more = false;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        store(0, i, cut_part(v[i]));
#pragma unroll
        for (int e = 0; e < 8; ++e) more |= v[i][e] != 0.f;
    }
    more = __syncthreads_or(more);
    if (threadIdx.x == 0) p.counts[blockIdx.x] = more ? MS_PARTS : 1;
    if (more)
#pragma unroll
        for (int q = 1; q < MS_PARTS; ++q)
#pragma unroll
            for (int i = 0; i < 2; ++i) store(q, i, cut_part(v[i]));
}

template <int BN>
static int split_launch(const void* a_parts, const void* w_parts, const SplitParams& p, cudaStream_t st, const char* what) {
    using Sh = SplitShape<BN>;
    static thread_local int configured_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (configured_dev != dev) {
        cudaError_t e = cudaFuncSetAttribute(mm_split_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Sh::SMEM_BYTES);
        if (e != cudaSuccess) return fail(BN_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
        configured_dev = dev;
    }
    CUtensorMap ma, mw;
    const uint64_t stride[1] = {(uint64_t)p.K * 2};
    const uint64_t dims_a[2] = {(uint64_t)p.K, (uint64_t)p.M * MS_PARTS}, dims_w[2] = {(uint64_t)p.K, (uint64_t)p.N * (p.counts ? MS_PARTS : p.w_parts)};
    const uint32_t box_a[2] = {MS_BK, MS_BM}, box_w[2] = {MS_BK, BN};
    if (int rc = make_tensor_map(&ma, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a_parts, dims_a, stride, box_a, CU_TENSOR_MAP_SWIZZLE_128B)) return rc;
    if (int rc = make_tensor_map(&mw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, w_parts, dims_w, stride, box_w, CU_TENSOR_MAP_SWIZZLE_128B)) return rc;
    const long long tiles = (long long)ceil_div(p.M, MS_BM) * ceil_div(p.N, BN);
    const int sms = sm_count();
    launch_dependent(mm_split_kernel<BN>, (unsigned)(tiles < sms ? tiles : sms), MS_THREADS, Sh::SMEM_BYTES, st, ma, mw, p);
    return launch_status(what);
}

// The tile width by an estimate of the time, in us: what 64 k of a tile take, measured with one tile per multiprocessor and with
// several (the same).  The tensor pipe is active 69 % of the time with three parts, 50 % with one, whose two stages do not cover
// the loads; L2 throughput a third of its peak.
// Products of 800 rows, chain (bn_mm_f32) / with operands cut, three parts / the same, one part: 2048 -> 7424 691 / 152 / 96 us,
// 2048 -> 2048 189 / 50 / 33 us, 7424 -> 2048 679 / 168 / 121 us; 64 rows 2048 -> 7424 81 / 60 / 38 us, 2048 -> 2048 34 / 39 / 26 us.
// (A stage with room for one part of the weight, three of them in flight or 256 columns wide, is no faster for one part - 107, 38,
// 119 us - and took 190, 64, 223 us for three.)
// Error against 64 bits (2-norms) at K = 2048: chain 8.1e-7, here 1.3e-7; at K = 7424 1.5e-6 and 2.1e-7.
static float split_estimate(int M, int N, int K, int w_nparts, int* bn) {
    const int sms = sm_count();
    float best = 0.f;
    for (int width = 64; width <= 128; width *= 2) {
        const long long tiles = (long long)ceil_div(M, MS_BM) * ceil_div(N, width);
        const float step = w_nparts == 1 ? (width == 64 ? 0.72f : 0.83f) : (width == 64 ? 1.2f : 1.42f);
        const float t = (float)((tiles + sms - 1) / sms) * (float)ceil_div(K, MS_BK) * step;
        if (width == 64 || t < best) {
            best = t;
            *bn = width;
        }
    }
    return best;
}

static int split_run(int bn, const void* a_parts, const void* w_parts, const SplitParams& p, cudaStream_t st, const char* what) {
    return bn == 128 ? split_launch<128>(a_parts, w_parts, p, st, what) : split_launch<64>(a_parts, w_parts, p, st, what);
}

}  // namespace bn

using namespace bn;

extern "C" int bn_split_f32(const float* x, int64_t ld, void* parts, int rows, int cols, bn_stream_t stream) {
    const char* what = "bn_split_f32";
    if (!x || !parts) return fail(BN_ERR_INVALID_ARG, "%s: null pointer", what);
    if (rows < 0 || cols < 0 || cols % 8 || ld % 4 || (reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(parts)) & 15)
        return fail(BN_ERR_INVALID_ARG, "%s: rows=%d cols=%d (a multiple of 8), 16-byte aligned rows", what, rows, cols);
    if (int rc = require_sm100()) return rc;
    const long long n = (long long)rows * cols / 8, blocks = (n + 255) / 256;
    if (n == 0) return BN_OK;
    split_parts_kernel<<<(unsigned)(blocks < 8192 ? blocks : 8192), 256, 0, as_stream(stream)>>>(
        x, ld, static_cast<__nv_bfloat16*>(parts), rows, cols);
    return launch_status(what);
}

extern "C" int bn_mm_f32_split(const void* a_parts, const void* w_parts, int w_nparts, const float* a, int64_t a_ld, const float* w,
                               int64_t w_ld, const float* bias, int act, float* c, int M, int N, int K, int* error_word,
                               bn_stream_t stream) {
    const char* what = "bn_mm_f32_split";
    if (!a_parts || !w_parts || !a || !w || !c) return fail(BN_ERR_INVALID_ARG, "%s: null pointer", what);
    if (M < 0 || N < 0 || K <= 0 || N % 8 || K % 8 || (w_nparts != 1 && w_nparts != MS_PARTS) || act < 0 || act > BN_ACT_LAST)
        return fail(BN_ERR_INVALID_ARG, "%s: bad shape M=%d N=%d K=%d parts=%d act=%d", what, M, N, K, w_nparts, act);
    if ((reinterpret_cast<uintptr_t>(c) | reinterpret_cast<uintptr_t>(bias)) & 15) return fail(BN_ERR_INVALID_ARG, "%s: alignment", what);
    if ((long long)M * MS_PARTS > INT32_MAX || (long long)N * MS_PARTS > INT32_MAX) return fail(BN_ERR_UNSUPPORTED, "%s: M=%d N=%d too large", what, M, N);
    if (int rc = require_sm100()) return rc;
    if (M == 0 || N == 0) return BN_OK;
    const bool aligned = ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w)) & 15) == 0 && a_ld % 4 == 0 && w_ld % 4 == 0;
    const SplitParams p{a, w, bias, c, error_word, nullptr, a_ld, w_ld, M, N, K, act, w_nparts, aligned};
    int bn;
    split_estimate(M, N, K, w_nparts, &bn);
    return split_run(bn, a_parts, w_parts, p, as_stream(stream), what);
}

// The cut operands of bn_linear_f32: parts of A, parts of the weight, counts of parts
struct CutLayout { size_t w_parts, counts, total; };
static CutLayout cut_layout(int M, int N, int K) {
    auto up = [](size_t n) { return (n + 255) & ~(size_t)255; };
    CutLayout l;
    l.w_parts = up((size_t)MS_PARTS * M * K * 2);
    l.counts = l.w_parts + up((size_t)MS_PARTS * N * K * 2);
    l.total = l.counts + (size_t)ceil_div(N, 64) * ceil_div(K, MS_BK);       // for the narrowest tiles
    return l;
}
static bool split_fits(int M, int N, int K) {
    return (long long)M * MS_PARTS <= INT32_MAX && (long long)N * MS_PARTS <= INT32_MAX &&
           (long long)ceil_div(N, 64) * ceil_div(K, MS_BK) < INT32_MAX - 8192;
}

extern "C" size_t bn_linear_f32_workspace_bytes(int M, int N, int K) { return M <= 0 || N <= 0 || K <= 0 ? 0 : cut_layout(M, N, K).total; }

// The time of bn_linear_f32: starts, the cut of the weight (6 or 10 bytes each) and of A, the product
static float parts_estimate(int M, int N, int K, int w_nparts, float product) {
    return 6.f + (float)N * (float)K * (w_nparts == 1 ? 0.8e-6f : 1.4e-6f) + (float)M * (float)K * 1.0e-6f + product;
}

// How a product is taken that bn_linear_f32_streams leaves (it has most of those of up to 16 rows, and many of up to 48), by estimates
// in us (measured, one part / three): operands cut, where that takes less time than bn_mm_f32; with up to 16 rows it does not, the
// weight being cut for them alone (2048 -> 32000, 4 / 16 / 32 rows: 169, 115, 114 / 251, 192, 192 us, chains 87, 100, 153).  Where the parts alone would have been faster (4 rows 108 us with the cut elsewhere, 16 rows 59), the
// weight is wide enough for bn_mm_f32_sums to hide its additions (4 / 12 rows 86.5 / 94.7 us, chains 86.5 / 91.9), and the error is
// the smaller one again; narrower weights, whose time is a chain's latency, keep the chains (1 x 2048 -> 2048 23.0 us, sums 27.1).
extern "C" int bn_linear_f32_form(int M, int N, int K, int w_nparts) {
    if (M <= 0 || N <= 0 || K <= 0 || N % 8 || K % 8 || !split_fits(M, N, K)) return BN_LINEAR_F32_CHAINS;
    int bn;
    const float product = split_estimate(M, N, K, w_nparts, &bn), chains = mm_f32_estimate(M, N, K);
    if (M > 16 && parts_estimate(M, N, K, w_nparts, product) < chains) return BN_LINEAR_F32_PARTS;
    return 11.f + (float)M * (float)K * 1.2e-6f + product < chains ? BN_LINEAR_F32_SUMS : BN_LINEAR_F32_CHAINS;
}

extern "C" int bn_linear_f32_streams(int M, int N, int K, int w_nparts) {
    if (M <= 0 || M > 48 || N <= 0 || K <= 0 || N % 8 || K % 8) return 0;      // (64 rows 2048 -> 2048: 32.3 us, chains 25.7)
    float other = mm_f32_estimate(M, N, K);
    if (M > 16 && split_fits(M, N, K)) {
        int bn;
        other = fminf(other, parts_estimate(M, N, K, w_nparts, split_estimate(M, N, K, w_nparts, &bn)));
    }
    return mm_stream_estimate(M, N, K) < other;
}

extern "C" int bn_linear_f32(const float* a, int64_t a_ld, const float* w, int64_t w_ld, const float* bias, int act, float* c, int M,
                             int N, int K, void* workspace, size_t workspace_bytes, int* error_word, bn_stream_t stream) {
    const char* what = "bn_linear_f32";
    if (!a || !w || !c) return fail(BN_ERR_INVALID_ARG, "%s: null pointer", what);
    if (M < 0 || N < 0 || K <= 0 || N % 8 || K % 8 || a_ld % 4 || w_ld % 4 || act < 0 || act > BN_ACT_LAST)
        return fail(BN_ERR_INVALID_ARG, "%s: bad shape M=%d N=%d K=%d act=%d", what, M, N, K, act);
    if ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(c) | reinterpret_cast<uintptr_t>(bias)) & 15)
        return fail(BN_ERR_INVALID_ARG, "%s: alignment", what);
    if (!split_fits(M, N, K)) return fail(BN_ERR_UNSUPPORTED, "%s: M=%d N=%d K=%d too large", what, M, N, K);
    if (int rc = require_sm100()) return rc;
    if (M == 0 || N == 0) return BN_OK;
    const CutLayout l = cut_layout(M, N, K);
    if (!workspace || reinterpret_cast<uintptr_t>(workspace) & 15 || workspace_bytes < l.total)
        return fail(BN_ERR_WORKSPACE, "%s: workspace of %zu bytes given, %zu needed, 16-byte aligned", what, workspace_bytes, l.total);
    uint8_t* ws = static_cast<uint8_t*>(workspace);
    cudaStream_t st = as_stream(stream);
    int bn;
    split_estimate(M, N, K, MS_PARTS, &bn);
    const long long n8 = (long long)M * K / 8, blocks_a = (n8 + bn * 4 - 1) / (bn * 4);
    const CutParams cp{a, w, reinterpret_cast<__nv_bfloat16*>(ws), reinterpret_cast<__nv_bfloat16*>(ws + l.w_parts), ws + l.counts, a_ld, w_ld, M, N,
                       K, ceil_div(N, bn) * ceil_div(K, MS_BK)};
    const unsigned grid = (unsigned)(cp.w_blocks + (blocks_a < 4096 ? blocks_a : 4096));
    if (bn == 64) launch_dependent(cut_operands_kernel<64>, grid, 256, 0, st, cp);
    else launch_dependent(cut_operands_kernel<128>, grid, 512, 0, st, cp);
    if (int rc = launch_status(what)) return rc;
    const SplitParams p{a, w, bias, c, error_word, cp.counts, a_ld, w_ld, M, N, K, act, 0, true};
    return split_run(bn, cp.a_parts, cp.w_parts, p, st, what);
}
