// fp32 path: operators whose arithmetic ORDER matches the reference's fp32 SIMT
// kernels, so that results agree with it far inside the 1e-5 gate instead of
// merely within rounding noise of the exact answer.
//
//   bn_rope_f32          reference: src/ops/op_rope.cuh:55-99
//   bn_attn_prefill_f32  rope -> q k^T -> *scale -> causal softmax -> p v fused
//                        in one launch, no (S,S) matrix in memory
//                        (reference sequence: mygrad/llama/llama_layers.py:161-183)
//
// These are parity kernels (small S, fp32); the roofline targets are the bf16
// kernels in attn_prefill_sm100.cu and attn_decode.cu.
#include "common.cuh"

namespace bn {

// ---------------------------------------------------------------------------
// RoPE, one thread per adjacent pair
// ---------------------------------------------------------------------------
__global__ void rope_f32_kernel(const float* __restrict__ x, int64_t x_rs, int64_t x_cs, float* __restrict__ y,
                                int64_t y_rs, int64_t y_cs, int rows, int cols, int head_dim, float theta,
                                int position_offset) {
    int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int pairs_per_row = cols / 2;
    if (idx >= (int64_t)rows * pairs_per_row) return;
    int row = (int)(idx / pairs_per_row);
    int c0 = (int)(idx % pairs_per_row) * 2;
    int pair = (c0 % head_dim) / 2;
    int position = row + position_offset;
    float freq = rope_inv_freq(pair, head_dim, theta);
    float angle = position * freq;
    float cos_angle = cosf(angle), sin_angle = sinf(angle);
    float x0 = x[row * x_rs + c0 * x_cs], x1 = x[row * x_rs + (c0 + 1) * x_cs];
    y[row * y_rs + c0 * y_cs] = x0 * cos_angle - x1 * sin_angle;
    y[row * y_rs + (c0 + 1) * y_cs] = x0 * sin_angle + x1 * cos_angle;
}

// ---------------------------------------------------------------------------
// Fused attention core, fp32
// ---------------------------------------------------------------------------
// A score is ONE chain of FMAs over the width of its softmax's problem (collapsed heads: all of Hq * D columns, 2048 links of
// 4 cycles = 4 us), an output one chain over the keys: the kernel is bound by those chains and by reading their operands from
// shared memory, so it spreads (row, key) pairs as widely as it can.  A CTA owns RPT x GR query rows of one problem; thread =
// (key of a 128-key tile, group of RPT rows).  The tile's rotated keys stay in shared memory for all the query heads that
// share them; queries are rotated in pieces of up to 256 columns.  Scores are kept (up to the shared memory that is left)
// and exponentiated once the row's maximum and sum are known, p = expf(s - m) / l; where they do not fit, they are
// computed twice, a tile at a time.
// 128 rows, 32 / 4 heads of 64, collapsed: 72 us; with 16 rows a CTA (8 CTAs) and all scores computed twice 699 us.
constexpr int AF_KEYS = 128, AF_QCOLS = 256;
constexpr int AF_MAXD = 64, AF_MAXOUT = 256;    // head_dim; distinct output columns of a problem
constexpr size_t AF_SMEM = 200 * 1024;

struct AttnF32Params {
    const float *q, *k, *v;
    float* out;
    int64_t q_rs, q_cs, k_rs, k_cs, v_rs, v_cs, o_rs, o_cs;
    int S, Hq, Hkv, D;
    float scale, theta;
    int position_offset, causal, heads_mode, apply_rope;
    int heads_per_piece, k_ld, p_ld, stored;
};

// PC: output columns of a problem, rounded up to 64 or 256.  D4: head_dim is a multiple of 4.
template <int RPT, int GR, int PC, bool D4>
__global__ void __launch_bounds__(AF_KEYS * GR) attn_f32_kernel(const AttnF32Params p) {
    constexpr int THREADS = AF_KEYS * GR, BM = RPT * GR;
    constexpr int CPT = PC > THREADS ? PC / THREADS : 1, NG = PC > THREADS ? 1 : THREADS / PC, ROWS = (BM + NG - 1) / NG;
    extern __shared__ __align__(16) float af_smem[];
    __shared__ float inv_freq[AF_MAXD / 2];
    __shared__ float row_m[BM], row_l[BM];
    float* Ks = af_smem;                                       // [key][k_ld]
    float* Qs = Ks + AF_KEYS * p.k_ld;                         // [row][heads_per_piece * D]
    float2* k_turn = reinterpret_cast<float2*>(Qs + BM * p.heads_per_piece * p.D);   // [key][D / 2] cos, sin
    float2* q_turn = k_turn + AF_KEYS * (p.D / 2);                                   // [row][D / 2]
    float* Ps = reinterpret_cast<float*>(q_turn + BM * (p.D / 2));                   // [row][p_ld]

    const int tid = threadIdx.x, key = tid % AF_KEYS, group = tid / AF_KEYS, warp = tid / 32, lane = tid % 32;
    const int D = p.D, half = D / 2, n_rep = p.Hq / p.Hkv, prob = blockIdx.y;
    const int row0 = (gridDim.x - 1 - blockIdx.x) * BM;        // the rows with most keys first
    const bool collapsed = p.heads_mode == BN_HEADS_COLLAPSED;
    const int heads = collapsed ? p.Hq : 1, kv_heads = collapsed ? p.Hkv : 1;
    const int head0 = collapsed ? 0 : prob, kv0 = collapsed ? 0 : prob / n_rep, Wo = kv_heads * D;
    const int last = p.causal ? min(p.S - 1, row0 + BM - 1 + p.position_offset) : p.S - 1;
    const int n_keys = last + 1, n_tiles = (n_keys + AF_KEYS - 1) / AF_KEYS;
    const int q_ld = p.heads_per_piece * D, pieces = (heads + p.heads_per_piece - 1) / p.heads_per_piece;

    if (tid < half) inv_freq[tid] = rope_inv_freq(tid, D, p.theta);
    if (tid < BM) { row_m[tid] = -INFINITY; row_l[tid] = 0.f; }
    __syncthreads();

    // cos and sin of rows g0 .. g0 + n - 1's positions
    auto turn = [&](int g0, int n, float2* cs) {
        if (!p.apply_rope) return;
        for (int e = tid; e < n * half; e += THREADS) {
            const float angle = (g0 + e / half + p.position_offset) * inv_freq[e % half];
            float cos_angle, sin_angle;
            sincosf(angle, &sin_angle, &cos_angle);
            cs[e] = make_float2(cos_angle, sin_angle);
        }
    };
    // rows [g0, g0 + n) of `heads_n` heads from `head_at` on, rotated, to dst[row][head * D ..]
    auto stage = [&](const float* x, int64_t rs, int64_t cs, int g0, int n, int head_at, int heads_n, const float2* turned, float* dst, int ld) {
        const int pairs = heads_n * half;
#pragma unroll 8
        for (int e = tid; e < n * pairs; e += THREADS) {
            const int r = e / pairs, c = e - r * pairs, i = c % half, g = g0 + r;
            float x0 = 0.f, x1 = 0.f;
            if (g < p.S) {
                const float* src = x + g * rs + (head_at * D + 2 * c) * cs;
                x0 = __ldg(src);
                x1 = __ldg(src + cs);
            }
            float y0 = x0, y1 = x1;
            if (p.apply_rope) {
                const float cos_angle = turned[r * half + i].x, sin_angle = turned[r * half + i].y;
                y0 = x0 * cos_angle - x1 * sin_angle;
                y1 = x0 * sin_angle + x1 * cos_angle;
            }
            *reinterpret_cast<float2*>(dst + r * ld + 2 * c) = make_float2(y0, y1);
        }
    };
    turn(row0, BM, q_turn);
    auto row_last = [&](int r) {
        const int g = row0 + r;
        return g >= p.S ? -1 : p.causal ? min(p.S - 1, g + p.position_offset) : p.S - 1;
    };
    // the tile's scaled scores to dst[row][key], -inf where masked
    auto scores = [&](int tile, float* dst) {
        const int j0 = tile * AF_KEYS;
        __syncthreads();                                       // the keys before, and what lies in dst, have been read
        turn(j0, AF_KEYS, k_turn);
        __syncthreads();
        stage(p.k, p.k_rs, p.k_cs, j0, AF_KEYS, kv0, kv_heads, k_turn, Ks, p.k_ld);
        float acc[RPT];
#pragma unroll
        for (int r = 0; r < RPT; ++r) acc[r] = 0.f;
        for (int piece = 0; piece < pieces; ++piece) {
            const int h0 = piece * p.heads_per_piece, nh = min(p.heads_per_piece, heads - h0);
            if (piece > 0) __syncthreads();                    // the queries before have been read
            if (pieces > 1 || tile == 0) stage(p.q, p.q_rs, p.q_cs, row0, BM, head0 + h0, nh, q_turn, Qs, q_ld);
            __syncthreads();
            for (int h = 0; h < nh; ++h) {
                const float* kr = Ks + key * p.k_ld + (collapsed ? (h0 + h) / n_rep * D : 0);
                const float* qr = Qs + group * RPT * q_ld + h * D;
                if (D4) {
#pragma unroll 4
                    for (int d = 0; d < D; d += 4) {
                        const float4 k4 = *reinterpret_cast<const float4*>(kr + d);
#pragma unroll
                        for (int r = 0; r < RPT; ++r) {
                            const float4 q4 = *reinterpret_cast<const float4*>(qr + r * q_ld + d);
                            acc[r] = fmaf(q4.w, k4.w, fmaf(q4.z, k4.z, fmaf(q4.y, k4.y, fmaf(q4.x, k4.x, acc[r]))));
                        }
                    }
                } else {
                    for (int d = 0; d < D; ++d)
#pragma unroll
                        for (int r = 0; r < RPT; ++r) acc[r] = fmaf(qr[r * q_ld + d], kr[d], acc[r]);
                }
            }
        }
        // scale: a separate fp32 multiply, as op_multiply does
#pragma unroll
        for (int r = 0; r < RPT; ++r)
            dst[(group * RPT + r) * p.p_ld + key] = j0 + key <= row_last(group * RPT + r) ? acc[r] * p.scale : -INFINITY;
    };
    // takes n scores of every row into its maximum and sum; a warp per row
    auto take = [&](const float* src, int n) {
        for (int r = warp; r < BM; r += THREADS / 32) {
            float m = row_m[r], sum = 0.f;
            for (int j = lane; j < n; j += 32) m = fmaxf(m, src[r * p.p_ld + j]);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            if (m > -INFINITY)
                for (int j = lane; j < n; j += 32) sum += expf(src[r * p.p_ld + j] - m);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            if (lane == 0 && m > -INFINITY) { row_l[r] = row_l[r] * expf(row_m[r] - m) + sum; row_m[r] = m; }
            __syncwarp();
        }
    };
    auto weights = [&](float* src, int j0, int n) {
        for (int e = tid; e < BM * n; e += THREADS) {
            const int r = e / n, j = e - r * n;
            float& s = src[r * p.p_ld + j];
            s = j0 + j <= row_last(r) ? expf(s - row_m[r]) / row_l[r] : 0.f;
        }
    };
    float out[ROWS][CPT];
#pragma unroll
    for (int i = 0; i < ROWS; ++i)
#pragma unroll
        for (int c = 0; c < CPT; ++c) out[i][c] = 0.f;
    const int col = tid % (PC / CPT), rg = tid / (PC / CPT);
    // out += the weights of keys j0 .. j0 + n - 1 times their values, in key order
    auto values = [&](const float* src, int j0, int n) {
#pragma unroll 16
        for (int j = 0; j < n; ++j) {
            float v[CPT];
#pragma unroll
            for (int c = 0; c < CPT; ++c)
                v[c] = col + c * (PC / CPT) < Wo ? __ldg(p.v + (int64_t)(j0 + j) * p.v_rs + (kv0 * D + col + c * (PC / CPT)) * p.v_cs) : 0.f;
#pragma unroll
            for (int i = 0; i < ROWS; ++i) {
                const int r = rg + i * NG;
                const float w = BM % NG == 0 || r < BM ? src[r * p.p_ld + j] : 0.f;
#pragma unroll
                for (int c = 0; c < CPT; ++c) out[i][c] = fmaf(w, v[c], out[i][c]);
            }
        }
    };

    if (p.stored) {
        for (int t = 0; t < n_tiles; ++t) scores(t, Ps + t * AF_KEYS);
        __syncthreads();
        take(Ps, n_keys);
        __syncthreads();
        weights(Ps, 0, n_keys);
        __syncthreads();
        values(Ps, 0, n_keys);
    } else {
        for (int t = 0; t < n_tiles; ++t) {
            scores(t, Ps);
            __syncthreads();
            take(Ps, AF_KEYS);
        }
        for (int t = 0; t < n_tiles; ++t) {
            const int n = min(AF_KEYS, n_keys - t * AF_KEYS);
            scores(t, Ps);
            __syncthreads();
            weights(Ps, t * AF_KEYS, n);
            __syncthreads();
            values(Ps, t * AF_KEYS, n);
        }
    }
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
        const int r = rg + i * NG, g = row0 + r;
        if (r >= BM || g >= p.S) continue;
#pragma unroll
        for (int c0 = 0; c0 < CPT; ++c0) {
            const int c = col + c0 * (PC / CPT);
            if (c >= Wo) continue;
            if (collapsed) {
                const int h = c / D, d = c - h * D;
                for (int rep = 0; rep < n_rep; ++rep) p.out[g * p.o_rs + ((h * n_rep + rep) * D + d) * p.o_cs] = out[i][c0];
            } else {
                p.out[g * p.o_rs + (prob * D + c) * p.o_cs] = out[i][c0];
            }
        }
    }
}

template <int RPT, int GR, int PC, bool D4>
static int attn_f32_run(AttnF32Params p, int problems, cudaStream_t st) {
    constexpr int BM = RPT * GR;
    const size_t fixed = (size_t)(AF_KEYS * p.k_ld + BM * p.heads_per_piece * p.D + (AF_KEYS + BM) * p.D) * sizeof(float);
    const int all_keys = ceil_div(p.S, AF_KEYS) * AF_KEYS + 4;
    p.stored = fixed + (size_t)BM * all_keys * sizeof(float) <= AF_SMEM;
    p.p_ld = p.stored ? all_keys : AF_KEYS + 4;
    const size_t smem = fixed + (size_t)BM * p.p_ld * sizeof(float);
    if (int rc = allow_smem(attn_f32_kernel<RPT, GR, PC, D4>, smem, "bn_attn_prefill_f32", SMEM_MOST, 512)) return rc;      // (its arrays: 144 - 256)
    attn_f32_kernel<RPT, GR, PC, D4><<<dim3(ceil_div(p.S, BM), problems), AF_KEYS * GR, smem, st>>>(p);
    return launch_status("bn_attn_prefill_f32");
}

template <int PC, bool D4>
static int attn_f32_rows(const AttnF32Params& p, int problems, cudaStream_t st) {
    // As many rows to a CTA as leave a CTA for every multiprocessor: rows share the keys' rotation and their reading from
    // shared memory, CTAs share nothing.
    const long long rows = (long long)p.S * problems, sms = sm_count();
    if (rows > 16 * sms / 2) return attn_f32_run<4, 4, PC, D4>(p, problems, st);
    if (rows > sms) return attn_f32_run<2, 2, PC, D4>(p, problems, st);
    return attn_f32_run<1, 1, PC, D4>(p, problems, st);
}

}  // namespace bn

using namespace bn;

extern "C" int bn_rope_f32(const float* x, int64_t x_rs, int64_t x_cs, float* y, int64_t y_rs, int64_t y_cs,
                           int rows, int cols, int head_dim, float theta, int position_offset,
                           bn_stream_t stream) {
    if (!x || !y) return fail(BN_ERR_INVALID_ARG, "bn_rope_f32: null pointer");
    if (rows < 0 || cols < 0 || head_dim <= 0 || head_dim % 2)
        return fail(BN_ERR_INVALID_ARG, "bn_rope_f32: bad shape rows=%d cols=%d head_dim=%d", rows, cols, head_dim);
    if (cols % head_dim != 0)
        return fail(BN_ERR_INVALID_ARG, "RoPE: hidden_dim must be divisible by head_dim");  // op_rope.cuh:115-117
    if (int rc = require_sm100()) return rc;
    int64_t n = (int64_t)rows * (cols / 2);
    if (n == 0) return BN_OK;
    rope_f32_kernel<<<(unsigned)((n + 255) / 256), 256, 0, as_stream(stream)>>>(x, x_rs, x_cs, y, y_rs, y_cs, rows,
                                                                               cols, head_dim, theta,
                                                                               position_offset);
    return launch_status("bn_rope_f32");
}

extern "C" int bn_attn_prefill_f32(const float* q, int64_t q_rs, int64_t q_cs, const float* k, int64_t k_rs,
                                   int64_t k_cs, const float* v, int64_t v_rs, int64_t v_cs, float* out,
                                   int64_t o_rs, int64_t o_cs, int S, int Hq, int Hkv, int D, float scale,
                                   float theta, int position_offset, int causal, int heads_mode, int apply_rope,
                                   bn_stream_t stream) {
    if (!q || !k || !v || !out) return fail(BN_ERR_INVALID_ARG, "bn_attn_prefill_f32: null pointer");
    if (S < 0 || Hq <= 0 || Hkv <= 0 || D <= 0)
        return fail(BN_ERR_INVALID_ARG, "bn_attn_prefill_f32: bad shape S=%d Hq=%d Hkv=%d D=%d", S, Hq, Hkv, D);
    if (Hq % Hkv != 0) return fail(BN_ERR_INVALID_ARG, "bn_attn_prefill_f32: Hq=%d not a multiple of Hkv=%d", Hq, Hkv);
    if (heads_mode != BN_HEADS_COLLAPSED && heads_mode != BN_HEADS_PER_HEAD)
        return fail(BN_ERR_INVALID_ARG, "bn_attn_prefill_f32: heads_mode=%d", heads_mode);
    if (D % 2 || D > AF_MAXD)
        return fail(BN_ERR_UNSUPPORTED, "bn_attn_prefill_f32: head_dim=%d (even, <= %d supported)", D, AF_MAXD);
    const int Wo = heads_mode == BN_HEADS_COLLAPSED ? Hkv * D : D;
    if (Wo > AF_MAXOUT)
        return fail(BN_ERR_UNSUPPORTED, "bn_attn_prefill_f32: Hkv*D=%d (<= %d supported)", Wo, AF_MAXOUT);
    if (int rc = require_sm100()) return rc;
    if (S == 0) return BN_OK;
    const int heads = heads_mode == BN_HEADS_COLLAPSED ? Hq : 1, problems = heads_mode == BN_HEADS_COLLAPSED ? 1 : Hq;
    const int per_piece = AF_QCOLS / D < heads ? AF_QCOLS / D : heads;
    // a row stride of 4 floats more than a multiple of 8 puts the 16-byte reads of eight neighbouring keys on different banks
    const int k_ld = (Wo + 7) / 8 * 8 + 4;
    const AttnF32Params p{q, k, v, out, q_rs, q_cs, k_rs, k_cs, v_rs, v_cs, o_rs, o_cs, S, Hq, Hkv, D,
                          scale, theta, position_offset, causal, heads_mode, apply_rope, per_piece, k_ld, 0, 0};
    cudaStream_t st = as_stream(stream);
    if (D % 4) return Wo <= 64 ? attn_f32_rows<64, false>(p, problems, st) : attn_f32_rows<256, false>(p, problems, st);
    return Wo <= 64 ? attn_f32_rows<64, true>(p, problems, st) : attn_f32_rows<256, true>(p, problems, st);
}
