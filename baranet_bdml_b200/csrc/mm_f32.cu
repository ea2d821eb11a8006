// fp32 matrix product in the reference's own arithmetic order: one FMA chain per output, k ascending (reference:
// src/ops/op_mm_optimized.cuh:35-62).
#include <math.h>

#include "common.cuh"
#include "hybrid.cuh"

namespace bn {

// ---------------------------------------------------------------------------
// GEMM.  Every output is ONE chain of K dependent FMAs, so neither K nor a chain can be split and small products are bound by
// the chain (4 cycles a link), large ones by the FMA pipes (128 per clock and multiprocessor).
//
// A tile of BM x BN outputs, TM x TN per thread.  Both operands lie in shared memory as they come from global memory, by
// cp.async: K-contiguous operands as rows of MM_K + 4 floats, an N-contiguous B as MM_K rows of BN columns.  A thread reads
// four k at a time of each of its rows (one 16-byte access); its rows are BM / TM apart, so that neighbouring threads read
// neighbouring rows, whose stride of 20 floats puts eight 16-byte accesses on 32 different banks.  Times: at mm_f32_pick.
// ---------------------------------------------------------------------------
constexpr int MM_K = 16, MM_LD = MM_K + 4, MM_STAGES = 4;

// Up to three products of one A in a launch (q, k and v of the attention layer: the two narrow ones alone leave most of the chip
// idle for as long as a chain takes): set s has the tile columns up to tile_end[s].
constexpr int MM_SETS = 3;
struct MmSet {
    const float* B;
    float* C;
    int64_t b_rs, b_cs, c_rs, c_cs;
    int N;
};
struct MmParams {
    const float* A;
    int64_t a_rs, a_cs;
    int M, K, sets;
    MmSet set[MM_SETS];
    int tile_end[MM_SETS];
};

// VA / VB: 16-byte copies along the operand's contiguous dimension (K for A; K for B, or N with B_N).  B_N: B lies in shared
// memory with N contiguous.
// SUMS: not one chain, but chains of 16 k, added up by eights, and these in a third sum: the error of K = 2048 falls from 8.1e-7 to
// 1.2e-7, of K = 7424 from 1.5e-6 to 1.7e-7 (2-norms, against 64 bits).  4 x 2048 -> 32000 86.5 us either way; where the time is the
// latency of few tiles the additions show: 1 x 2048 -> 2048 23.0 us, sums 27.1; 4 x 7424 -> 2048 108.9 and 115.3.  (Chains of 16 in
// one sum 24.9 us and 2.2e-7, chains of 64 27.7 us and 1.8e-7.)
template <int BM, int BN, int TM, int TN, bool VA, bool VB, bool B_N, bool SUMS>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
mm_f32_kernel(const __grid_constant__ MmParams p) {
    constexpr int THREADS = (BM / TM) * (BN / TN), ROWS_T = BM / TM, COLS_T = BN / TN;
    constexpr int A_FLOATS = BM * MM_LD, B_FLOATS = B_N ? MM_K * BN : BN * MM_LD, STAGE = A_FLOATS + B_FLOATS;
    constexpr bool B_N4 = B_N && TN % 4 == 0;              // a thread's columns in groups of four neighbours
    extern __shared__ __align__(16) float mm_smem[];
    const uint32_t smem = ptx::smem_u32(mm_smem);
    const int tid = threadIdx.x, tx = tid % COLS_T, ty = tid / COLS_T;
    const int tile = blockIdx.x, s = (tile >= p.tile_end[0]) + (tile >= p.tile_end[1]);
    const MmSet& q = p.set[s];
    const int row0 = blockIdx.y * BM, col0 = (tile - (s ? p.tile_end[s - 1] : 0)) * BN;
    const int steps = (p.K + MM_K - 1) / MM_K;

    // What lies outside the operands becomes zero: a chain's last links then add 0 * 0.  16-byte copies go from a source of the
    // thread's own that advances by a step (null: a row or column outside).
    constexpr int NA = (BM * (MM_K / 4) + THREADS - 1) / THREADS, NB = (BN * (MM_K / 4) + THREADS - 1) / THREADS;
    const float *src_a[NA], *src_b[NB];
    uint32_t dst_a[NA], dst_b[NB];
    int k_a[NA], k_b[NB];
    if (VA) {
#pragma unroll
        for (int i = 0; i < NA; ++i) {
            const int e = tid + i * THREADS, r = e / (MM_K / 4), k = e % (MM_K / 4) * 4;
            src_a[i] = r < BM && row0 + r < p.M ? p.A + (row0 + r) * p.a_rs + k : nullptr;
            dst_a[i] = r < BM ? smem + (r * MM_LD + k) * 4 : 0;
            k_a[i] = k;
        }
    }
    if (VB) {
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            const int e = tid + i * THREADS, c = B_N ? e % (BN / 4) * 4 : e / (MM_K / 4), k = B_N ? e / (BN / 4) : e % (MM_K / 4) * 4;
            const bool mine = e < BN * (MM_K / 4);
            src_b[i] = mine && col0 + c < q.N ? q.B + (B_N ? k * q.b_rs + col0 + c : (col0 + c) * q.b_cs + k) : nullptr;
            dst_b[i] = mine ? smem + (A_FLOATS + (B_N ? k * BN + c : c * MM_LD + k)) * 4 : 0;
            k_b[i] = k;
        }
    }
    const int64_t advance_b = B_N ? MM_K * q.b_rs : MM_K;
    auto stage_in = [&](int step) {
        const uint32_t at = (step % MM_STAGES) * (STAGE * 4);
        const int k0 = step * MM_K;
        if (VA) {
#pragma unroll
            for (int i = 0; i < NA; ++i)
                if ((BM * (MM_K / 4)) % THREADS == 0 || dst_a[i]) {
                    const bool in = src_a[i] && k0 + k_a[i] < p.K;
                    ptx::cp_async_16(dst_a[i] + at, in ? src_a[i] : p.A, in ? 16 : 0);
                    if (src_a[i]) src_a[i] += MM_K;
                }
        } else {
            for (int e = tid; e < BM * MM_K; e += THREADS) {
                const int r = e / MM_K, k = e % MM_K;
                const bool in = row0 + r < p.M && k0 + k < p.K;
                ptx::cp_async_4(smem + at + (r * MM_LD + k) * 4, p.A + (in ? (row0 + r) * p.a_rs + (k0 + k) * p.a_cs : 0), in ? 4 : 0);
            }
        }
        if (VB) {
#pragma unroll
            for (int i = 0; i < NB; ++i)
                if ((BN * (MM_K / 4)) % THREADS == 0 || dst_b[i]) {
                    const bool in = src_b[i] && k0 + k_b[i] < p.K;
                    ptx::cp_async_16(dst_b[i] + at, in ? src_b[i] : q.B, in ? 16 : 0);
                    if (src_b[i]) src_b[i] += advance_b;
                }
        } else {
            for (int e = tid; e < BN * MM_K; e += THREADS) {
                const int c = e / MM_K, k = e % MM_K;
                const bool in = col0 + c < q.N && k0 + k < p.K;
                ptx::cp_async_4(smem + at + (A_FLOATS + c * MM_LD + k) * 4, q.B + (in ? (k0 + k) * q.b_rs + (col0 + c) * q.b_cs : 0),
                                in ? 4 : 0);
            }
        }
    };

    float acc[TM][TN], eights[TM][TN], total[TM][TN];
    // SUMS: takes a sum into the next one
    auto fold = [](float (&from)[TM][TN], float (&into)[TM][TN]) {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                into[i][j] += from[i][j];
                from[i][j] = 0.f;
            }
    };
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = eights[i][j] = total[i][j] = 0.f;

    // the operands of four k: b[column][k], or with B_N4 b[column group * 4 + k][column of the group]
    struct Frag { float a[TM][4], b[TN][4]; };
    auto load_frag = [&](Frag& f, int step, int k) {
        const float* sa = mm_smem + (step % MM_STAGES) * STAGE;
        const float* sb = sa + A_FLOATS;
#pragma unroll
        for (int i = 0; i < TM; ++i) load4(sa + (ty + i * ROWS_T) * MM_LD + k, f.a[i]);
        if (B_N4) {
#pragma unroll
            for (int j = 0; j < TN / 4; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) load4(sb + (k + e) * BN + (tx + j * COLS_T) * 4, f.b[j * 4 + e]);
        } else if (B_N) {
#pragma unroll
            for (int j = 0; j < TN; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) f.b[j][e] = sb[(k + e) * BN + tx + j * COLS_T];
        } else {
#pragma unroll
            for (int j = 0; j < TN; ++j) load4(sb + (tx + j * COLS_T) * MM_LD + k, f.b[j]);
        }
    };

#pragma unroll
    for (int s = 0; s < MM_STAGES; ++s) {
        if (s < steps) stage_in(s);
        ptx::cp_async_commit();
    }
    // Fragments are read a group of four k ahead of their use, across the steps' ends: few warps share a scheduler, and a
    // shared-memory round trip in front of every group would stand open.
    Frag f[2];
    ptx::cp_async_wait<MM_STAGES - 1>();
    __syncthreads();
    load_frag(f[0], 0, 0);
    for (int step = 0; step < steps; ++step) {
#pragma unroll
        for (int g = 0; g < MM_K / 4; ++g) {
            if (g == MM_K / 4 - 1) {
                ptx::cp_async_wait<MM_STAGES - 2>();
                __syncthreads();                           // the next step's tiles are there, and this step's have been read
                if (step + MM_STAGES < steps) stage_in(step + MM_STAGES);
                ptx::cp_async_commit();
                load_frag(f[(g + 1) & 1], step + 1, 0);    // (behind the last step: read and not used)
            } else {
                load_frag(f[(g + 1) & 1], step, (g + 1) * 4);
            }
            const Frag& c = f[g & 1];
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j)
                        acc[i][j] = fmaf(c.a[i][e], B_N4 ? c.b[j / 4 * 4 + e][j % 4] : c.b[j][e], acc[i][j]);
        }
        if (SUMS) {
            fold(acc, eights);
            if (step % 8 == 7) fold(eights, total);
        }
    }
    if (SUMS) fold(eights, total);
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int r = row0 + ty + i * ROWS_T;
        if (r >= p.M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int c = col0 + (B_N4 ? (tx + j / 4 * COLS_T) * 4 + j % 4 : tx + j * COLS_T);
            if (c < q.N) q.C[r * q.c_rs + c * q.c_cs] = SUMS ? total[i][j] : acc[i][j];
        }
    }
}

template <int BM, int BN, int TM, int TN, bool VA, bool VB, bool B_N, bool SUMS>
static int mm_f32_run(MmParams p, cudaStream_t st) {
    constexpr size_t smem = (size_t)MM_STAGES * (BM * MM_LD + (B_N ? MM_K * BN : BN * MM_LD)) * sizeof(float);
    if (int rc = allow_smem(mm_f32_kernel<BM, BN, TM, TN, VA, VB, B_N, SUMS>, smem, "bn_mm_f32")) return rc;
    for (int s = 0; s < MM_SETS; ++s) p.tile_end[s] = (s ? p.tile_end[s - 1] : 0) + (s < p.sets ? ceil_div(p.set[s].N, BN) : 0);
    const dim3 grid(p.tile_end[MM_SETS - 1], ceil_div(p.M, BM));
    if (grid.y > 65535) return fail(BN_ERR_UNSUPPORTED, "bn_mm_f32: M=%d too large", p.M);
    mm_f32_kernel<BM, BN, TM, TN, VA, VB, B_N, SUMS><<<grid, (BM / TM) * (BN / TN), smem, st>>>(p);
    return launch_status("bn_mm_f32");
}

// How the operands can be copied: A and B along K, B along N, 16 bytes at a time where the strides and addresses allow it.
template <int BM, int BN, int TM, int TN, bool SUMS>
static int mm_f32_copies(const MmParams& p, cudaStream_t st) {
    auto fours = [](const float* x, int64_t contiguous, int64_t other, int n) {
        return contiguous == 1 && other % 4 == 0 && n % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
    };
    const bool va = fours(p.A, p.a_cs, p.a_rs, p.K);
    bool along_n = va, along_k = va;                       // every set's B
    for (int s = 0; s < p.sets; ++s) {
        along_n = along_n && fours(p.set[s].B, p.set[s].b_cs, p.set[s].b_rs, p.set[s].N);
        along_k = along_k && fours(p.set[s].B, p.set[s].b_rs, p.set[s].b_cs, p.K);
    }
    if constexpr (!SUMS)
        if (along_n) return mm_f32_run<BM, BN, TM, TN, true, true, true, SUMS>(p, st);
    if (along_k) return mm_f32_run<BM, BN, TM, TN, true, true, false, SUMS>(p, st);
    return mm_f32_run<BM, BN, TM, TN, false, false, false, SUMS>(p, st);
}

// The tile by an estimate of the time: a tile alone on a multiprocessor takes `alone` (its chains' latency), several there take
// `more` each (the pipes).  Both in us at K = 2048, measured: one tile per multiprocessor, and M = 800 with N = 4608 .. 7424.
// Small tiles spread a small product over the chip, large ones read shared memory less often; what bounds the large ones is
// that reading (8 x 4 outputs a thread: 12 16-byte reads, 4 cycles each, for 128 FMAs), 53 - 60 % of the FMA rate.
// One 64 x 64 tile of 4 x 4 outputs a thread without copies in flight, before / after: 128 x 2048 x 2048 134 / 52 us,
// 128 x 256 x 2048 134 / 24 us, 800 x 7424 x 2048 1470 / 610 us, 4 x 32000 x 2048 570 / 88 us.
// sums: without the largest tile, whose threads have no registers for three sums
static float mm_f32_times(int M, const int* N, int sets, bool sums, int* best) {
    const int sms = sm_count();
    auto estimate = [&](int bm, int bn, float alone, float more) {
        long long tiles = 0;
        for (int s = 0; s < sets; ++s) tiles += (long long)ceil_div(M, bm) * ceil_div(N[s], bn);
        if (ceil_div(M, bm) > 65535 && bm < 128) return INFINITY;        // the grid's limit
        return fmaxf(alone, (float)((tiles + sms - 1) / sms) * more);
    };
    const float t[5] = {estimate(128, 128, 221.f, 220.f), estimate(64, 64, 77.f, 62.f), estimate(32, 64, 52.f, 34.f),
                        estimate(16, 32, 33.f, 16.f), estimate(8, 32, 24.f, 10.4f)};
    *best = sums ? 1 : 0;
    for (int i = *best + 1; i < 5; ++i)
        if (t[i] < t[*best]) *best = i;
    return t[*best];
}

template <bool SUMS>
static int mm_f32_pick(const MmParams& p, cudaStream_t st) {
    int best, n[MM_SETS];
    for (int s = 0; s < p.sets; ++s) n[s] = p.set[s].N;
    mm_f32_times(p.M, n, p.sets, SUMS, &best);
    switch (best) {
        case 0:
            if constexpr (!SUMS) return mm_f32_copies<128, 128, 8, 8, false>(p, st);
        case 1: return mm_f32_copies<64, 64, 8, 4, SUMS>(p, st);
        case 2: return mm_f32_copies<32, 64, 4, 4, SUMS>(p, st);
        case 3: return mm_f32_copies<16, 32, 4, 2, SUMS>(p, st);
        default: return mm_f32_copies<8, 32, 2, 1, SUMS>(p, st);
    }
}

float mm_f32_estimate(int M, int N, int K) {
    int best;
    return mm_f32_times(M, &N, 1, false, &best) * (float)K / 2048.f;
}

// x = act(x + bias) in place, fp32 rows (the unfused form of the products with a bias or an activation)
__global__ void __launch_bounds__(256)
bias_act_kernel(float* x, int64_t ld, const float* bias, long long n, int cols, int act) {
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < n; i += (long long)gridDim.x * 256) {
        const int64_t r = i / cols, c = i - r * cols;
        x[r * ld + c] = activation_exact(act, x[r * ld + c] + (bias ? bias[c] : 0.f));
    }
}

}  // namespace bn

using namespace bn;

extern "C" int bn_mm_f32(const float* A, int64_t a_rs, int64_t a_cs, const float* B, int64_t b_rs, int64_t b_cs,
                         float* C, int64_t c_rs, int64_t c_cs, int M, int K, int N, bn_stream_t stream) {
    if (!A || !B || !C) return fail(BN_ERR_INVALID_ARG, "bn_mm_f32: null pointer");
    if (M < 0 || K < 0 || N < 0) return fail(BN_ERR_INVALID_ARG, "bn_mm_f32: negative size");
    if (int rc = require_sm100()) return rc;
    if (M == 0 || N == 0) return BN_OK;
    MmParams p{A, a_rs, a_cs, M, K, 1, {{B, C, b_rs, b_cs, c_rs, c_cs, N}}, {}};
    return mm_f32_pick<false>(p, as_stream(stream));
}

extern "C" int bn_mm_f32_sums(const float* a, int64_t a_ld, const float* w, int64_t w_ld, float* c, int64_t c_ld, int M, int N, int K,
                              bn_stream_t stream) {
    if (!a || !w || !c) return fail(BN_ERR_INVALID_ARG, "bn_mm_f32_sums: null pointer");
    if (M < 0 || K < 0 || N < 0) return fail(BN_ERR_INVALID_ARG, "bn_mm_f32_sums: negative size");
    if (int rc = require_sm100()) return rc;
    if (M == 0 || N == 0) return BN_OK;
    MmParams p{a, a_ld, 1, M, K, 1, {{w, c, 1, w_ld, c_ld, 1, N}}, {}};
    if (ceil_div(M, 64) > 65535) return mm_f32_pick<false>(p, as_stream(stream));      // the grid's limit
    return mm_f32_pick<true>(p, as_stream(stream));
}

extern "C" int bn_mm_f32_each(const float* A, int64_t a_rs, int64_t a_cs, int n, const float* const* B, const int64_t* b_rs,
                              const int64_t* b_cs, float* const* C, const int64_t* c_rs, const int64_t* c_cs, int M, int K, const int* N,
                              bn_stream_t stream) {
    const char* what = "bn_mm_f32_each";
    if (!A || !B || !b_rs || !b_cs || !C || !c_rs || !c_cs || !N) return fail(BN_ERR_INVALID_ARG, "%s: null pointer", what);
    if (n < 0 || n > MM_SETS || M < 0 || K < 0) return fail(BN_ERR_INVALID_ARG, "%s: bad shape n=%d M=%d K=%d", what, n, M, K);
    MmParams p{A, a_rs, a_cs, M, K, 0, {}, {}};
    for (int s = 0; s < n; ++s) {
        if (!B[s] || !C[s] || N[s] < 0) return fail(BN_ERR_INVALID_ARG, "%s: product %d", what, s);
        if (N[s] > 0) p.set[p.sets++] = MmSet{B[s], C[s], b_rs[s], b_cs[s], c_rs[s], c_cs[s], N[s]};
    }
    if (int rc = require_sm100()) return rc;
    if (M == 0 || p.sets == 0) return BN_OK;
    return mm_f32_pick<false>(p, as_stream(stream));
}

extern "C" int bn_bias_act_f32(float* x, int64_t ld, const float* bias, int rows, int cols, int act, bn_stream_t stream) {
    if (!x) return fail(BN_ERR_INVALID_ARG, "bn_bias_act_f32: null pointer");
    if (rows < 0 || cols < 0 || act < 0 || act > BN_ACT_LAST) return fail(BN_ERR_INVALID_ARG, "bn_bias_act_f32: bad shape or activation");
    if (int rc = require_sm100()) return rc;
    const long long n = (long long)rows * cols;
    if (n == 0) return BN_OK;
    const long long blocks = (n + 255) / 256;
    bias_act_kernel<<<(unsigned)(blocks < 4096 ? blocks : 4096), 256, 0, as_stream(stream)>>>(x, ld, bias, n, cols, act);
    return launch_status("bn_bias_act_f32");
}
