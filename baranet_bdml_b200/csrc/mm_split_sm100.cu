// fp32 products of many rows on the tensor cores: C (M,N) = act(A (M,K) W (N,K)^T + bias), both operands cut into bf16 parts.
//
// A 24-bit significand is three bf16 numbers: x1 = bf16(x), x2 = bf16(x - x1), x3 = x - x1 - x2, exactly.  Of the nine products
// of parts the six down to 2^-18 of the largest are taken; the three left out are below 2^-26 of |a b|, less than the rounding
// of a partial sum of an fp32 chain.  A weight that is a bf16 number (a bf16 checkpoint run in fp32) has one part, and three
// products are all there are.
//
// The tensor cores add into fp32 accumulators with truncation, which over a long K would cost more than a chain of FMAs does.
// So an accumulator takes 64 k only, the small products first and x1 w1 last, and these sums are added up in registers, rounded
// to nearest: 4 truncations at full size in an accumulator, K / 64 roundings in a sum, where a chain has K.
//
// An element whose sum is not finite (an infinity or a NaN among the operands, a part that overflows bf16, a sum that does) is
// worked out again as a chain of FMAs from the fp32 operands.
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

// WP: parts of the weight (1 or 3)
template <int BN, int WP> struct SplitShape {
    static constexpr int A_BYTES = MS_BM * MS_BK * 2, B_BYTES = BN * MS_BK * 2;
    static constexpr int STAGE_BYTES = MS_PARTS * A_BYTES + WP * B_BYTES;
    static constexpr int NSTAGE = 204800 / STAGE_BYTES;
    static constexpr int SMEM_BYTES = 1024 + NSTAGE * STAGE_BYTES;
    static constexpr uint32_t TMEM_COLS = 2 * BN;
};

struct SplitParams {
    const float *a, *w, *bias;
    float* c;
    int* error_word;
    int64_t a_ld, w_ld;
    int M, N, K, act;
};

template <int BN, int WP>
__global__ void __launch_bounds__(MS_THREADS, 1)
mm_split_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_w, const SplitParams p) {
    using Sh = SplitShape<BN, WP>;
    constexpr int NSTAGE = Sh::NSTAGE;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bar_full[NSTAGE], bar_empty[NSTAGE], bar_acc_full[2], bar_acc_empty[2];
    __shared__ uint32_t s_tmem_base;
    __shared__ int s_abort;

    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int tiles_m = (p.M + MS_BM - 1) / MS_BM, tiles_n = (p.N + BN - 1) / BN, n_tiles = tiles_m * tiles_n;
    const int k_steps = (p.K + MS_BK - 1) / MS_BK;

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

    if (warp == 9) {
        if (lane == 0) {
            prefetch_tensormap(&tmap_a);
            prefetch_tensormap(&tmap_w);
            uint32_t it = 0;
            bool ok = true;
            for (int t = blockIdx.x; ok && t < n_tiles; t += gridDim.x) {
                const int m0 = t % tiles_m * MS_BM, n0 = t / tiles_m * BN;
                for (int ks = 0; ks < k_steps; ++ks, ++it) {
                    const int stage = it % NSTAGE;
                    ok = mbar_wait(smem_u32(&bar_empty[stage]), ((it / NSTAGE) & 1u) ^ 1u, &s_abort);
                    if (!ok) break;
                    const uint32_t full = smem_u32(&bar_full[stage]), sA = smem0 + stage * Sh::STAGE_BYTES, sW = sA + MS_PARTS * Sh::A_BYTES;
                    mbar_arrive_expect_tx(full, Sh::STAGE_BYTES);
                    // part q of A is rows q M .. q M + M - 1 of its map: a tile's rows beyond M are rows that are not stored
#pragma unroll
                    for (int q = 0; q < MS_PARTS; ++q) tma_load_2d(sA + q * Sh::A_BYTES, &tmap_a, ks * MS_BK, q * p.M + m0, full);
#pragma unroll
                    for (int q = 0; q < WP; ++q) tma_load_2d(sW + q * Sh::B_BYTES, &tmap_w, ks * MS_BK, q * p.N + n0, full);
                }
            }
        }
    } else if (warp == 8) {
        constexpr uint32_t IDESC = tc::idesc_bf16(MS_BM, BN, 0);
        const uint64_t d0 = tc::smem_desc_sw128(0);
        // (part of A, part of W), the smallest products first
        constexpr int PRODUCTS = WP == 1 ? 3 : 6;
        constexpr int PA[6] = {2, WP == 1 ? 1 : 0, WP == 1 ? 0 : 1, 1, 0, 0}, PW[6] = {0, WP == 1 ? 0 : 2, WP == 1 ? 0 : 1, 0, 1, 0};
        uint32_t it = 0;
        bool ok = true;
        for (int t = blockIdx.x; ok && t < n_tiles; t += gridDim.x) {
            for (int ks = 0; ks < k_steps; ++ks, ++it) {
                const uint32_t acc = it & 1u, stage = it % NSTAGE;
                ok = mbar_wait(smem_u32(&bar_acc_empty[acc]), ((it >> 1) & 1u) ^ 1u, &s_abort) &&
                     mbar_wait(smem_u32(&bar_full[stage]), (it / NSTAGE) & 1u, &s_abort);
                if (!ok) break;
                if (elect_one()) {
                    tc::fence_after_sync();
                    const uint32_t s0 = smem0 + stage * Sh::STAGE_BYTES;
#pragma unroll
                    for (int q = 0; q < PRODUCTS; ++q) {
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
            if (gm < p.M) {
                float* crow = p.c + (size_t)gm * p.N + n0;
                const bool late = p.act != BN_ACT_NONE && p.act != BN_ACT_RELU2;
#pragma unroll
                for (int c = 0; c < COLS / 32; ++c) {
                    bool bad = false;
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
                    if (bad || late)
#pragma unroll 1
                        for (int k = c * 32; k < c * 32 + 32 && n0 + k < p.N; ++k) {
                            float s = crow[k];
                            if (bad) {
                                const float *x = p.a + gm * p.a_ld, *y = p.w + (n0 + k) * p.w_ld;
                                s = 0.f;
#pragma unroll 1
                                for (int i = 0; i < p.K; ++i) s = fmaf(x[i], y[i], s);
                                if (p.bias) s += p.bias[n0 + k];
                            }
                            crow[k] = activation_exact(p.act, s);
                        }
                }
            }
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

// x (rows, cols) -> parts [3][rows][cols]; cols a multiple of 8.  What is not finite in bf16 stays in the first part alone.
__global__ void __launch_bounds__(256)
split_parts_kernel(const float* x, int64_t ld, __nv_bfloat16* parts, long long rows, int cols) {
    const long long n8 = rows * (cols / 8), plane = rows * cols;
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < n8; i += (long long)gridDim.x * 256) {
        const long long r = i / (cols / 8);
        const float* s = x + r * ld + (i - r * (cols / 8)) * 8;
        float v[8];
        load4(s, *reinterpret_cast<float(*)[4]>(v));
        load4(s + 4, *reinterpret_cast<float(*)[4]>(v + 4));
#pragma unroll
        for (int q = 0; q < MS_PARTS; ++q) {
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                w[e] = pack_bf16(v[2 * e], v[2 * e + 1]);
                const float lo = bf16_lo(w[e]), hi = bf16_hi(w[e]);
                v[2 * e] = fabsf(lo) <= FLT_MAX ? v[2 * e] - lo : 0.f;
                v[2 * e + 1] = fabsf(hi) <= FLT_MAX ? v[2 * e + 1] - hi : 0.f;
            }
            *reinterpret_cast<uint4*>(parts + q * plane + i * 8) = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
}

template <int BN, int WP>
static int split_launch(const void* a_parts, const void* w_parts, const SplitParams& p, cudaStream_t st) {
    using Sh = SplitShape<BN, WP>;
    const char* what = "bn_mm_f32_split";
    static thread_local int configured_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (configured_dev != dev) {
        cudaError_t e = cudaFuncSetAttribute(mm_split_kernel<BN, WP>, cudaFuncAttributeMaxDynamicSharedMemorySize, Sh::SMEM_BYTES);
        if (e != cudaSuccess) return fail(BN_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
        configured_dev = dev;
    }
    CUtensorMap ma, mw;
    const uint64_t stride[1] = {(uint64_t)p.K * 2};
    const uint64_t dims_a[2] = {(uint64_t)p.K, (uint64_t)p.M * MS_PARTS}, dims_w[2] = {(uint64_t)p.K, (uint64_t)p.N * WP};
    const uint32_t box_a[2] = {MS_BK, MS_BM}, box_w[2] = {MS_BK, BN};
    if (int rc = make_tensor_map(&ma, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a_parts, dims_a, stride, box_a, CU_TENSOR_MAP_SWIZZLE_128B)) return rc;
    if (int rc = make_tensor_map(&mw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, w_parts, dims_w, stride, box_w, CU_TENSOR_MAP_SWIZZLE_128B)) return rc;
    const long long tiles = (long long)ceil_div(p.M, MS_BM) * ceil_div(p.N, BN);
    const int sms = sm_count();
    mm_split_kernel<BN, WP><<<(unsigned)(tiles < sms ? tiles : sms), MS_THREADS, Sh::SMEM_BYTES, st>>>(ma, mw, p);
    return launch_status(what);
}

// The tile width by an estimate of the time, in us: what 64 k of a tile take, measured with one tile per multiprocessor and with
// several (the same: a tile's loads and MMAs both read or write shared memory, 96 - 290 KB in this time).  128 x 256 does not fit
// twice with three parts of the weight.  The start and the parts of A (bn_split_f32) come on top.
// Products of 800 rows, chain (bn_mm_f32) / three parts / one part, the 8 - 15 us of bn_split_f32 not counted:
// 2048 -> 7424 664 / 130 / 84 us, 2048 -> 2048 180 / 49 / 31 us, 7424 -> 2048 621 / 143 / 85 us; 64 rows 2048 -> 7424 82 / 46 / 27 us.
// Error against 64 bits (2-norms) at K = 2048: chain 8.1e-7, here 1.3e-7; at K = 7424 1.5e-6 and 2.1e-7.
static float split_estimate(int M, int N, int K, int w_nparts, int* bn) {
    const int sms = sm_count();
    const float steps = (float)ceil_div(K, MS_BK);
    float best = 0.f;
    for (int width = 64; width <= (w_nparts == 1 ? 256 : 128); width *= 2) {
        const long long tiles = (long long)ceil_div(M, MS_BM) * ceil_div(N, width);
        const float step = w_nparts == 1 ? (width == 64 ? 0.72f : width == 128 ? 0.88f : 1.42f) : (width == 64 ? 1.2f : 1.42f);
        const float t = (float)((tiles + sms - 1) / sms) * steps * step;
        if (width == 64 || t < best) {
            best = t;
            *bn = width;
        }
    }
    return 11.f + (float)M * (float)K * 1.2e-6f + best;
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
    const SplitParams p{a, w, bias, c, error_word, a_ld, w_ld, M, N, K, act};
    int bn;
    split_estimate(M, N, K, w_nparts, &bn);
    cudaStream_t st = as_stream(stream);
    if (w_nparts == 1) {
        if (bn == 256) return split_launch<256, 1>(a_parts, w_parts, p, st);
        return bn == 128 ? split_launch<128, 1>(a_parts, w_parts, p, st) : split_launch<64, 1>(a_parts, w_parts, p, st);
    }
    return bn == 128 ? split_launch<128, 3>(a_parts, w_parts, p, st) : split_launch<64, 3>(a_parts, w_parts, p, st);
}

extern "C" int bn_mm_f32_split_pays(int M, int N, int K, int w_nparts) {
    if (M <= 0 || N <= 0 || K <= 0 || (long long)M * MS_PARTS > INT32_MAX || (long long)N * MS_PARTS > INT32_MAX) return 0;
    int bn;
    return split_estimate(M, N, K, w_nparts, &bn) < mm_f32_estimate(M, N, K);
}
