// The fp32 attention layer in one call: q, k, v projections, RoPE, causal softmax attention (collapsed heads or one softmax per
// query head) and the output projection (reference sequence: mygrad/llama/llama_layers.py:155-186).
//
// Collapsed heads have ONE softmax over the scores summed over all query heads.  The reps query heads that share a key head meet
// the same keys, at the same rotation, so  sum_h rot(q_h) . rot(k) = rot(sum_h q_h) . rot(k),  and a sum of heads is a product
// with the sum of their weight columns; the reps output heads are one and the same, so the output projection reads them with the
// sum of its weight rows.  32 query heads over 4 key heads of 64: 2048 columns of q, of every score and of the output
// projection's K become 256.  The weights are summed in the call (reading them is what the
// layer cannot do without); every sum is fp32, and shorter than the one it replaces.
//
// 128 rows, width 2048, 32 / 4 heads of 64, collapsed: 41 us; as four operators (three products in a launch, scores of 2048 columns,
// output projection of K = 2048) 215 us.  Error against 64 bits (2-norm) 6e-7, before 3.8e-6; so the distance to the reference's own
// chains is 4e-6 (2e-6 to 6e-6 over lengths), where the four operators differ from them in the order of the softmax sum alone.  Per head
// 109 us, before 158 us.  Products are of bf16 parts, which hold an fp32 number exactly from 2^-109 on and what lies below to 2^-134.
//
//   0 fold_kernel (collapsed)   the query weight's columns summed        3 attention over rotated rows
//   1 project_kernel            x @ [Wq | Wk | Wv] over ranges of k      4 out_kernel (collapsed), or project_kernel + add_ranges_kernel
//   2 finish_kernel             the ranges added up, q and k rotated; beside it (collapsed) the output weight's rows summed
#include <float.h>

#include "attn_portion.cuh"
#include "common.cuh"
#include "hybrid.cuh"
#include "ptx.cuh"

namespace bn {

constexpr int AL_THREADS = 256, AL_KEYS = 64, AL_MAXW = 256, AL_MAXD = 64;
constexpr size_t AL_SMEM = SMEM_MOST;

__device__ __forceinline__ float4 add4(const float4& a, const float4& b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

// The sum of the `reps` groups of four floats that lie `stride` apart, past L1: a weight may have been written since L1 read it.
// Pairs first: log2(reps) roundings instead of reps.
__device__ __forceinline__ float4 sum_heads(const float* at, int64_t stride, int reps) {
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    int r = 0;
    for (; r + 8 <= reps; r += 8) {
        float4 v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = __ldcg(reinterpret_cast<const float4*>(at + (r + i) * stride));
        s = add4(s, add4(add4(add4(v[0], v[1]), add4(v[2], v[3])), add4(add4(v[4], v[5]), add4(v[6], v[7]))));
    }
    for (; r < reps; ++r) s = add4(s, __ldcg(reinterpret_cast<const float4*>(at + r * stride)));
    return s;
}

// fp32 numbers as three bf16 parts each, x = hi + mid + lo (mm_split_sm100.cu has the bounds), pairs packed
struct Parts { uint32_t p[3]; };
__device__ __forceinline__ Parts cut(float x, float y) {
    Parts r;
    r.p[0] = ptx::pack_bf16(x, y);
    x -= ptx::bf16_lo(r.p[0]); y -= ptx::bf16_hi(r.p[0]);
    r.p[1] = ptx::pack_bf16(x, y);
    r.p[2] = ptx::pack_bf16(x - ptx::bf16_lo(r.p[1]), y - ptx::bf16_hi(r.p[1]));
    return r;
}
// the six products of parts down to 2^-18 of the largest, the largest last: (part of A, part of B)
#define BN_PART_PRODUCTS constexpr int PART_A[6] = {2, 0, 1, 1, 0, 0}, PART_B[6] = {0, 2, 1, 0, 1, 0}

// ---- 0: w (hidden, groups * reps * D) -> (hidden, groups * D), a thread per four columns
__global__ void __launch_bounds__(AL_THREADS) fold_kernel(const float* w, int64_t w_rs, float* out, int hidden, int groups, int reps, int D) {
    const int quads = groups * D / 4;
    const long long n = (long long)hidden * quads;
    ptx::grid_dependency_wait();
    ptx::grid_launch_dependents();
    for (long long e = (long long)blockIdx.x * AL_THREADS + threadIdx.x; e < n; e += (long long)gridDim.x * AL_THREADS) {
        const int row = (int)(e / quads), c = (int)(e % quads) * 4;
        *reinterpret_cast<float4*>(out + (int64_t)row * (quads * 4) + c) = sum_heads(w + row * w_rs + (int64_t)(c / D) * reps * D + c % D, D, reps);
    }
}

// ---- 1: C[z] = A[:, range z] @ B[range z, :], as products of bf16 parts on warp-level tensor cores.
// A block has BM rows, 64 columns and a range of k, which it walks in chunks of 32: a thread loads 8 k of a row of A and 512 / BM
// numbers of B two chunks ahead, cuts them a chunk ahead and leaves the parts in shared memory, two stages.  A warp has 32 x 16
// outputs; a chunk is 48 MMAs of it (8 cycles each a scheduler, 0.8 us a chunk of 128 rows).  The tensor cores add with truncation, so
// an accumulator takes 32 k, the small products first, and is then added up in registers.
// fp32 FMAs are bound by reading shared memory here (8 x 4 outputs a thread, or 4 x 4): 128 rows, 2048 -> 256 + 256 + 256, 18 - 20 us;
// this one 15 us.  Error of the sums, K = 2048: as mm_split_kernel's, 1.3e-7.
// An infinity, or a number whose bf16 rounding overflows, makes NaN of its sums: what is not finite is worked out again as a chain.
constexpr int PJ_BN = 64, PJ_KC = 32, PJ_SETS = 3, PJ_A_LD = PJ_KC + 8, PJ_B_LD = PJ_BN + 8;
struct ProjectSet {
    const float* B;
    int64_t b_rs;
    int N;
};
struct ProjectParams {
    const float* A;
    int64_t a_rs;
    float* C;                    // [ranges][M][ld]
    int M, K, ld, range, sets;
    ProjectSet set[PJ_SETS];
    int tile_end[PJ_SETS];
};

// neither an infinity nor a NaN
__device__ __forceinline__ bool finite(float v) { return fabsf(v) <= FLT_MAX; }

template <int BM>
__global__ void __launch_bounds__(BM * 4, 1) project_kernel(const __grid_constant__ ProjectParams p) {
    constexpr int THREADS = BM * 4, QB = PJ_KC * PJ_BN / 4 / THREADS;      // quads of B a thread has of a chunk
    constexpr int A_PART = BM * PJ_A_LD, B_PART = PJ_KC * PJ_B_LD, STAGE = 3 * (A_PART + B_PART);
    BN_PART_PRODUCTS;
    extern __shared__ __align__(16) __nv_bfloat16 pj_smem[];
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32, tile = blockIdx.x;
    const int s = (tile >= p.tile_end[0]) + (tile >= p.tile_end[1]);
    const ProjectSet& q = p.set[s];
    const int n0 = (tile - (s ? p.tile_end[s - 1] : 0)) * PJ_BN, row0 = blockIdx.y * BM;
    const int k0 = blockIdx.z * p.range, kn = min(p.K - k0, p.range), chunks = (kn + PJ_KC - 1) / PJ_KC;
    const uint32_t smem = ptx::smem_u32(pj_smem);
    // this thread's part of a chunk: 8 k of row a_row of A, and quad tid % 16 of rows b_k + (THREADS / 16) i of B
    const int a_row = tid / 4, a_k = tid % 4 * 8, b_k = tid / 16, b_c = tid % 16 * 4;
    const bool a_in = row0 + a_row < p.M, b_in = n0 + b_c < q.N;
    const float* a_at = p.A + (a_in ? (row0 + a_row) * p.a_rs : 0) + k0 + a_k;
    const float* b_at = q.B + (int64_t)(k0 + b_k) * q.b_rs + (b_in ? n0 + b_c : 0);
    struct Piece { float4 a[2], b[QB]; } near, far;            // a chunk's and the one's behind it
    auto load = [&](Piece& t, int c) {                         // K and the range are multiples of 4; what lies outside becomes zero
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 2; ++i) t.a[i] = a_in && c * PJ_KC + a_k + i * 4 < kn ? *reinterpret_cast<const float4*>(a_at + c * PJ_KC + i * 4) : zero;
#pragma unroll
        for (int i = 0; i < QB; ++i) {
            const int k = c * PJ_KC + i * (THREADS / 16);
            t.b[i] = b_in && k + b_k < kn ? *reinterpret_cast<const float4*>(b_at + (int64_t)k * q.b_rs) : zero;
        }
    };
    auto store = [&](const Piece& t, int c) {
        __nv_bfloat16* sa = pj_smem + (c & 1) * STAGE;
        __nv_bfloat16* sb = sa + 3 * A_PART;
        const Parts x0 = cut(t.a[0].x, t.a[0].y), x1 = cut(t.a[0].z, t.a[0].w), x2 = cut(t.a[1].x, t.a[1].y), x3 = cut(t.a[1].z, t.a[1].w);
#pragma unroll
        for (int e = 0; e < 3; ++e)
            *reinterpret_cast<uint4*>(sa + e * A_PART + a_row * PJ_A_LD + a_k) = make_uint4(x0.p[e], x1.p[e], x2.p[e], x3.p[e]);
#pragma unroll
        for (int i = 0; i < QB; ++i) {
            const Parts y0 = cut(t.b[i].x, t.b[i].y), y1 = cut(t.b[i].z, t.b[i].w);
#pragma unroll
            for (int e = 0; e < 3; ++e)
                *reinterpret_cast<uint2*>(sb + e * B_PART + (b_k + i * (THREADS / 16)) * PJ_B_LD + b_c) = make_uint2(y0.p[e], y1.p[e]);
        }
    };
    ptx::grid_dependency_wait();
    ptx::grid_launch_dependents();
    load(near, 0);
    load(far, 1);
    const int wm = warp / 4 * 32, wn = warp % 4 * 16;          // the warp's outputs inside the tile
    float total[2][2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) total[i][j][0] = total[i][j][1] = total[i][j][2] = total[i][j][3] = 0.f;
    store(near, 0);
    near = far;
    load(far, 2);
    for (int c = 0; c < chunks; ++c) {
        __syncthreads();                                       // chunk c is there, and the stage of chunk c + 1 has been read
        if (c + 1 < chunks) {
            store(near, c + 1);
            near = far;
            load(far, c + 3);
        }
        const uint32_t ua = smem + (c & 1) * STAGE * 2 + ((wm + lane % 16) * PJ_A_LD + lane / 16 * 8) * 2;
        const uint32_t ub = smem + ((c & 1) * STAGE + 3 * A_PART) * 2 + (lane % 16 * PJ_B_LD + wn + lane / 16 * 8) * 2;
        float acc[2][2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.f;
        auto multiply = [&](const uint32_t (&x)[2][4], const uint32_t (&y)[4]) {
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) ptx::mma_bf16_16816(acc[i][j], x[i][0], x[i][1], x[i][2], x[i][3], y[2 * j], y[2 * j + 1]);
        };
        auto frag_a = [&](int part, int ks, uint32_t (&x)[2][4]) {
#pragma unroll
            for (int i = 0; i < 2; ++i) ptx::ldmatrix_x4(ua + (part * A_PART + i * 16 * PJ_A_LD + ks * 16) * 2, x[i][0], x[i][1], x[i][2], x[i][3]);
        };
        auto frag_b = [&](int part, int ks, uint32_t (&y)[4]) { ptx::ldmatrix_x4_trans(ub + (part * B_PART + ks * 16 * PJ_B_LD) * 2, y[0], y[1], y[2], y[3]); };
        uint32_t x[3][2][4], y[3][4];
#pragma unroll
        for (int ks = 0; ks < PJ_KC / 16; ++ks) {
#pragma unroll
            for (int e = 0; e < 3; ++e) { frag_a(e, ks, x[e]); frag_b(e, ks, y[e]); }
#pragma unroll
            for (int t = 0; t < 5; ++t) multiply(x[PART_A[t]], y[PART_B[t]]);
        }
#pragma unroll
        for (int ks = PJ_KC / 16 - 1; ks >= 0; --ks) {
            if (ks < PJ_KC / 16 - 1) { frag_a(0, ks, x[0]); frag_b(0, ks, y[0]); }
            multiply(x[0], y[0]);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) total[i][j][e] += acc[i][j][e];
    }
    int col0 = n0 + wn;                                        // the sets' columns lie side by side
    for (int i = 0; i < s; ++i) col0 += p.set[i].N;
    float* out = p.C + (int64_t)blockIdx.z * p.M * p.ld;
    // (row, column) of the sum in total[i][j][2 h + e]
    const int r0 = row0 + wm + lane / 4, c0 = lane % 4 * 2;
    // a sum that is not finite, as a chain
    auto chain = [&](int r, int n) {
        float sum = 0.f;
        for (int k = k0; k < k0 + kn; ++k) sum = fmaf(p.A[r * p.a_rs + k], q.B[k * q.b_rs + n], sum);
        return sum;
    };
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = r0 + i * 16 + h * 8;
            if (r >= p.M) continue;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int n = n0 + wn + j * 8 + c0;
                if (n >= q.N) continue;                        // N is a multiple of 4
                float2 v = make_float2(total[i][j][2 * h], total[i][j][2 * h + 1]);
                if (!finite(v.x)) v.x = chain(r, n);
                if (!finite(v.y)) v.y = chain(r, n + 1);
                *reinterpret_cast<float2*>(out + (int64_t)r * p.ld + col0 + j * 8 + c0) = v;
            }
        }
}

// ---- 2
struct FinishParams {
    const float* part;           // [ranges][S][Wq + 2 Wk]
    float* rows;                 // [S][Wq + 2 Wk]: rotated q | rotated k | v
    int ranges, S, Wq, Wk, D, offset;
    float theta;
    const float* wo;             // collapsed: the output weight (reps * Wq, hidden)
    float* wo_sums;              // (Wq, hidden)
    int64_t wo_rs;
    int hidden, reps;
};

// A block per row: the angles of its position are worked out once.  Blocks from S on sum the output weight's rows, which only the last
// launch reads: that stream runs beside the latencies of the rotation and of the attention.  (`wo` is as old as the call, whose first
// launch has waited for what wrote it; so is what read `wo_sums` before.)
__global__ void __launch_bounds__(AL_THREADS) finish_kernel(const FinishParams p) {
    __shared__ float2 turn[AL_MAXD / 2];
    const int tid = threadIdx.x, half = p.D / 2, ld = p.Wq + 2 * p.Wk;
    const int row = blockIdx.x;
    if (row >= p.S) {
        const int quads = p.hidden / 4;
        const long long n = (long long)p.Wq * quads, step = (long long)(gridDim.x - p.S) * AL_THREADS;
        for (long long e = (long long)(row - p.S) * AL_THREADS + tid; e < n; e += step) {
            const int r = (int)(e / quads), c = (int)(e % quads) * 4;
            *reinterpret_cast<float4*>(p.wo_sums + (int64_t)r * p.hidden + c) =
                sum_heads(p.wo + ((int64_t)(r / p.D) * p.reps * p.D + r % p.D) * p.wo_rs + c, (int64_t)p.D * p.wo_rs, p.reps);
        }
    } else if (tid < half) {
        const float angle = (row + p.offset) * rope_inv_freq(tid, p.D, p.theta);
        float cos_angle, sin_angle;
        sincosf(angle, &sin_angle, &cos_angle);
        turn[tid] = make_float2(cos_angle, sin_angle);
    }
    __syncthreads();
    ptx::grid_dependency_wait();
    ptx::grid_launch_dependents();
    const int64_t range = (int64_t)p.S * ld;
    for (int c = tid * 4; c < ld && row < p.S; c += AL_THREADS * 4) {
        const float* at = p.part + (int64_t)row * ld + c;
        float4 s = *reinterpret_cast<const float4*>(at);
#pragma unroll 12
        for (int z = 1; z < p.ranges; ++z) s = add4(s, *reinterpret_cast<const float4*>(at + z * range));
        if (c < p.Wq + p.Wk) {
            const float2 t0 = turn[c % p.D / 2], t1 = turn[c % p.D / 2 + 1];
            s = make_float4(s.x * t0.x - s.y * t0.y, s.x * t0.y + s.y * t0.x, s.z * t1.x - s.w * t1.y, s.z * t1.y + s.w * t1.x);
        }
        *reinterpret_cast<float4*>(p.rows + (int64_t)row * ld + c) = s;
    }
}

// ---- 4 (per head): sums of ranges, in order
__global__ void __launch_bounds__(AL_THREADS) add_ranges_kernel(const float* part, float* out, int64_t out_rs, int rows, int cols, int ranges) {
    const int quads = cols / 4;
    const long long n = (long long)rows * quads;
    ptx::grid_dependency_wait();
    ptx::grid_launch_dependents();
    for (long long e = (long long)blockIdx.x * AL_THREADS + threadIdx.x; e < n; e += (long long)gridDim.x * AL_THREADS) {
        const int r = (int)(e / quads), c = (int)(e % quads) * 4;
        const float* at = part + (int64_t)r * cols + c;
        float4 s = *reinterpret_cast<const float4*>(at);
#pragma unroll 4
        for (int z = 1; z < ranges; ++z) s = add4(s, *reinterpret_cast<const float4*>(at + z * (int64_t)rows * cols));
        *reinterpret_cast<float4*>(out + r * out_rs + c) = s;
    }
}

// ---- 3: attention over rotated rows.  A block owns BM query rows of one problem (collapsed: the only one, W = Hkv D columns; per
// head: W = D); tiles of 64 keys by cp.async, two in flight.  Four threads share a key, each takes its groups of four columns in turn for all BM rows (with the row stride of
// W + 16 floats eight neighbouring threads read 32 banks).  The scores stay in shared memory; a warp per row takes its maximum and
// sum, p = expf(s - m) / l.  Values: a thread has four columns and every n-th key for all BM rows, read as they come from L2, as
// many at a time as there are registers for; the n sums are added up in shared memory.
struct CoreParams {
    const float* rows;           // [S][ld]: q | k | v
    float* out;                  // [S][problems * W]
    int S, ld, k_at, v_at, W, problems, reps, p_ld;
    float scale;
    int offset, causal;
};

template <int BM>
__global__ void __launch_bounds__(AL_THREADS) attn_rows_f32_kernel(const CoreParams p) {
    constexpr int KEYS = AL_KEYS;
    extern __shared__ __align__(16) float al_smem[];
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32, W = p.W, k_ld = W + 16, quads = W / 4;
    const int prob = blockIdx.y, row0 = (gridDim.x - 1 - blockIdx.x) * BM;           // the rows with most keys first
    float* Ks = al_smem;                                                             // [2][KEYS][k_ld]
    float* Qs = Ks + 2 * KEYS * k_ld;                                             // [BM][W]
    float* Ps = Qs + BM * W;                                                         // [BM][p_ld]
    const float* q = p.rows + prob * W;
    const float* k = p.rows + p.k_at + prob / p.reps * W;
    const float* v = p.rows + p.v_at + prob / p.reps * W;
    auto row_last = [&](int r) {
        const int g = row0 + r;
        return g >= p.S ? -1 : p.causal ? min(p.S - 1, g + p.offset) : p.S - 1;
    };
    const int n_keys = (p.causal ? min(p.S - 1, row0 + BM - 1 + p.offset) : p.S - 1) + 1, tiles = (n_keys + KEYS - 1) / KEYS;
    const uint32_t uK = ptx::smem_u32(Ks), uQ = ptx::smem_u32(Qs);
    ptx::grid_dependency_wait();
    ptx::grid_launch_dependents();
    const int parts = AL_THREADS / quads, c4 = tid % quads, vp = tid / quads;          // a thread's four columns, of every parts-th row
    auto ask_keys = [&](int t) {
        if (t < tiles && vp < parts)
            for (int r = vp; r < KEYS; r += parts) {
                const bool in = t * KEYS + r < p.S;
                ptx::cp_async_16(uK + (((t & 1) * KEYS + r) * k_ld + c4 * 4) * 4, k + (in ? (int64_t)(t * KEYS + r) * p.ld + c4 * 4 : 0), in ? 16 : 0);
            }
        ptx::cp_async_commit();
    };
    for (int r = vp; r < BM && vp < parts; r += parts) {
        const bool in = row0 + r < p.S;
        ptx::cp_async_16(uQ + (r * W + c4 * 4) * 4, q + (in ? (int64_t)(row0 + r) * p.ld + c4 * 4 : 0), in ? 16 : 0);
    }
    ask_keys(0);
    ask_keys(1);
    constexpr int SHARE = AL_THREADS / KEYS;
    const int key = tid / SHARE, part = tid % SHARE;
    for (int t = 0; t < tiles; ++t) {
        ptx::cp_async_wait<1>();
        __syncthreads();
        float acc[BM];
#pragma unroll
        for (int r = 0; r < BM; ++r) acc[r] = 0.f;
        const float* kr = Ks + ((t & 1) * KEYS + key) * k_ld;
#pragma unroll 4
        for (int c = part * 4; c < W; c += SHARE * 4) {
            const float4 k4 = *reinterpret_cast<const float4*>(kr + c);
#pragma unroll
            for (int r = 0; r < BM; ++r) {
                const float4 q4 = *reinterpret_cast<const float4*>(Qs + r * W + c);
                acc[r] = fmaf(q4.w, k4.w, fmaf(q4.z, k4.z, fmaf(q4.y, k4.y, fmaf(q4.x, k4.x, acc[r]))));
            }
        }
#pragma unroll
        for (int r = 0; r < BM; ++r) {
#pragma unroll
            for (int o = 1; o < SHARE; o <<= 1) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], o);
            if (part == r % SHARE) Ps[r * p.p_ld + t * KEYS + key] = t * KEYS + key <= row_last(r) ? acc[r] * p.scale : -INFINITY;
        }
        __syncthreads();                                       // the tile has been read
        ask_keys(t + 2);
    }
    ptx::cp_async_wait_all();
    // keys up to `all` are seen by all the rows; few rows leave registers to ask for a thread's first values ahead of the softmax
    constexpr int AHEAD = BM <= 2 ? 16 : 1;
    const int all = row0 + BM <= p.S ? row_last(0) : -1;
    const float* vc = v + c4 * 4;
    float4 early[AHEAD];
    if (AHEAD > 1)
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
            const int j = vp + i * parts;
            early[i] = vp < parts && j <= all ? *reinterpret_cast<const float4*>(vc + (int64_t)j * p.ld) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    __syncthreads();
    for (int r = warp; r < BM; r += AL_THREADS / 32) {
        float* s = Ps + r * p.p_ld;
        float m = -INFINITY, l = 0.f;
        for (int j = lane; j < n_keys; j += 32) m = fmaxf(m, s[j]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        const int last = row_last(r);
        for (int j = lane; j < n_keys; j += 32) {
            // (a row that sees no key, or scores that are all -inf: as in attn_f32_kernel, whose sum stays 0)
            const float e = j <= last && m > -INFINITY ? expf(s[j] - m) : 0.f;
            s[j] = j <= last && !(m > -INFINITY) ? s[j] - m : e;
            l += e;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
        for (int j = lane; j < n_keys; j += 32)
            if (j <= last) s[j] = s[j] / l;
    }
    __syncthreads();
    float4 acc[BM];
#pragma unroll
    for (int r = 0; r < BM; ++r) acc[r] = make_float4(0.f, 0.f, 0.f, 0.f);
    auto take = [&](int r, int j, const float4& v4) {
        const float w = Ps[r * p.p_ld + j];
        acc[r].x = fmaf(w, v4.x, acc[r].x);
        acc[r].y = fmaf(w, v4.y, acc[r].y);
        acc[r].z = fmaf(w, v4.z, acc[r].z);
        acc[r].w = fmaf(w, v4.w, acc[r].w);
    };
    if (vp < parts) {
        int j = vp;
        if (AHEAD > 1) {
#pragma unroll
            for (int i = 0; i < AHEAD; ++i)
                if (vp + i * parts <= all) {
#pragma unroll
                    for (int r = 0; r < BM; ++r) take(r, vp + i * parts, early[i]);
                    j += parts;
                }
        }
#pragma unroll 8
        for (; j <= all; j += parts) {
            const float4 v4 = *reinterpret_cast<const float4*>(vc + (int64_t)j * p.ld);
#pragma unroll
            for (int r = 0; r < BM; ++r) take(r, j, v4);
        }
        for (; j < n_keys; j += parts) {                       // (left out, not multiplied by 0: a value may not be finite)
            const float4 v4 = *reinterpret_cast<const float4*>(vc + (int64_t)j * p.ld);
#pragma unroll
            for (int r = 0; r < BM; ++r)
                if (j <= row_last(r)) take(r, j, v4);
        }
    }
    // the sums of the parts, in order: over the keys' tiles (read by now), as many rows at a time as fit
    float4* sums = reinterpret_cast<float4*>(Ks);
    const int fit = 2 * KEYS * k_ld / (parts * W);
    for (int r0 = 0; r0 < BM; r0 += fit) {
        if (vp < parts)
#pragma unroll
            for (int r = 0; r < BM; ++r)
                if (r >= r0 && r < r0 + fit) sums[((r - r0) * parts + vp) * quads + c4] = acc[r];
        __syncthreads();
        const int n = min(fit, BM - r0) * quads;
        for (int e = tid; e < n; e += AL_THREADS) {
            const int r = r0 + e / quads, c = e % quads;
            float4 s = sums[((r - r0) * parts) * quads + c];
            for (int i = 1; i < parts; ++i) s = add4(s, sums[((r - r0) * parts + i) * quads + c]);
            if (row0 + r < p.S) *reinterpret_cast<float4*>(p.out + (int64_t)(row0 + r) * (p.problems * W) + prob * W + c * 4) = s;
        }
        __syncthreads();
    }
}

// ---- 4 (collapsed): out = attn (S, W) @ w, the summed rows of the output weight, by parts as above.  A block has 16 rows a warp and 16
// columns; it cuts its part of the weight before it waits for the attention (the sums were left two launches earlier, and the launch
// between has waited for that one).  A warp's rows go from global memory into its fragments, all of 128 k at a time.
// 128 rows, W = 256, 2048 columns: 8 us behind the attention; as fp32 FMAs 10 us.
constexpr int OUT_BN = 16, OUT_LD = OUT_BN + 8, OUT_AHEAD = 8;
struct OutParams {
    const float* attn;           // [S][W]
    const float* w;              // [W][hidden]
    float* out;
    int64_t out_rs;
    int S, W, hidden;
};

template <int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 1) out_kernel(const OutParams p) {
    BN_PART_PRODUCTS;
    extern __shared__ __align__(16) __nv_bfloat16 out_smem[];  // [part][K][24], K = W rounded up to 16
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32, col0 = blockIdx.x * OUT_BN, steps = (p.W + 15) / 16, PART = steps * 16 * OUT_LD;
    const int wr0 = (blockIdx.y * WARPS + warp) * 16;
    {
        const int c = tid % 4 * 4, col = col0 + c;
#pragma unroll 4
        for (int k = tid / 4; k < steps * 16; k += WARPS * 8) {
            const float4 v = col < p.hidden && k < p.W ? __ldcg(reinterpret_cast<const float4*>(p.w + (int64_t)k * p.hidden + col))
                                                       : make_float4(0.f, 0.f, 0.f, 0.f);
            const Parts y0 = cut(v.x, v.y), y1 = cut(v.z, v.w);
#pragma unroll
            for (int e = 0; e < 3; ++e) *reinterpret_cast<uint2*>(out_smem + e * PART + k * OUT_LD + c) = make_uint2(y0.p[e], y1.p[e]);
        }
    }
    ptx::grid_dependency_wait();
    ptx::grid_launch_dependents();
    // rows g and g + 8 of the warp's 16, k 2 j, 2 j + 1 and those 8 on of each 16: the A fragment of a step
    const int g = lane / 4, j = lane % 4;
    const float* a_at = p.attn + (int64_t)(wr0 + g) * p.W + 2 * j;
    const bool in0 = wr0 + g < p.S, in1 = wr0 + g + 8 < p.S;
    float2 av[OUT_AHEAD][4];
    auto load = [&](float2 (&v)[4], int ks) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {                          // (row, half of the step) = (e % 2, e / 2), as the fragment has them
            const bool in = (e % 2 ? in1 : in0) && ks * 16 + e / 2 * 8 + 2 * j < p.W;      // W is a multiple of 4
            v[e] = in ? *reinterpret_cast<const float2*>(a_at + (int64_t)(e % 2 * 8) * p.W + ks * 16 + e / 2 * 8) : make_float2(0.f, 0.f);
        }
    };
#pragma unroll
    for (int i = 0; i < OUT_AHEAD; ++i) load(av[i], i);
    __syncthreads();
    float total[2][4] = {}, small[2][4] = {}, big[2][4] = {};
    const uint32_t ub = ptx::smem_u32(out_smem) + (lane % 16 * OUT_LD + lane / 16 * 8) * 2;
    for (int ks0 = 0; ks0 < steps; ks0 += OUT_AHEAD) {
#pragma unroll
        for (int i = 0; i < OUT_AHEAD; ++i) {
            const int ks = ks0 + i;
            if (ks < steps) {
                Parts x[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) x[e] = cut(av[i][e].x, av[i][e].y);
                if (ks + OUT_AHEAD < steps) load(av[i], ks + OUT_AHEAD);
                uint32_t y[3][4];
#pragma unroll
                for (int e = 0; e < 3; ++e) ptx::ldmatrix_x4_trans(ub + (e * PART + ks * 16 * OUT_LD) * 2, y[e][0], y[e][1], y[e][2], y[e][3]);
#pragma unroll
                for (int t = 0; t < 6; ++t)
#pragma unroll
                    for (int n = 0; n < 2; ++n)
                        ptx::mma_bf16_16816(t < 5 ? small[n] : big[n], x[0].p[PART_A[t]], x[1].p[PART_A[t]], x[2].p[PART_A[t]], x[3].p[PART_A[t]],
                                            y[PART_B[t]][2 * n], y[PART_B[t]][2 * n + 1]);
            }
        }
#pragma unroll
        for (int n = 0; n < 2; ++n)                            // an accumulator takes 128 k, the small products one of their own
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                total[n][e] += small[n][e] + big[n][e];
                small[n][e] = big[n][e] = 0.f;
            }
    }
    auto chain = [&](int r, int col) {                         // a sum that is not finite
        float sum = 0.f;
        for (int k = 0; k < p.W; ++k) sum = fmaf(p.attn[(int64_t)r * p.W + k], p.w[(int64_t)k * p.hidden + col], sum);
        return sum;
    };
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int r = wr0 + g + h * 8;
        if (r >= p.S) continue;
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            const int col = col0 + n * 8 + 2 * j;
            if (col >= p.hidden) continue;                     // a multiple of 4
            float2 v = make_float2(total[n][2 * h], total[n][2 * h + 1]);
            if (!finite(v.x)) v.x = chain(r, col);
            if (!finite(v.y)) v.y = chain(r, col + 1);
            *reinterpret_cast<float2*>(p.out + r * p.out_rs + col) = v;
        }
    }
}

// allow_smem, asked of the driver once per thread and device for each kernel: what it sets does not depend on the call
template <auto KERNEL>
static int allow_smem_once(size_t bytes) {
    static thread_local int known_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (bytes <= 48 * 1024 || dev == known_dev) return BN_OK;
    if (int rc = allow_smem(KERNEL, bytes, "bn_attn_layer_f32")) return rc;
    known_dev = dev;
    return BN_OK;
}

struct LayerPlan {
    int Wq, Wk, W, problems, reps, ld, in_bm, in_range, out_bm, out_range, BM, wanted, p_ld;
    bool collapsed, fold, tiled;
    size_t wq_at, wo_at, part_at, rows_at, attn_at, out_at, total, smem;
};

// Rows to a block, and how K is cut: whole rounds of blocks, as many to a multiprocessor as their threads and shared memory allow,
// each of which takes about 2 us and, as long as it has the multiprocessor to itself, 1 us a chunk of 32 k and 128 rows.  A range is
// a write and a read of the result more.
static void project_plan(int M, int tiles, int K, int* bm, int* range) {
    const int sms = sm_count();
    *bm = M > 64 ? 128 : M > 32 ? 64 : 32;
    const long long blocks = (long long)tiles * ceil_div(M, *bm);
    float least = 1e30f;
    for (int n = 1; n <= 32 && (n == 1 || K / n >= PJ_KC); ++n) {
        const int r = ceil_div(ceil_div(K, n), PJ_KC) * PJ_KC, ranges = ceil_div(K, r);
        const long long busy = (blocks * ranges + sms - 1) / sms;          // blocks that the busiest multiprocessor has
        const float t = 2.f * ((busy + 1) / 2) + busy * (r / PJ_KC) * (0.3f + *bm / 180.f) + 6e-7f * M * tiles * PJ_BN * ranges;
        if (t < least) { least = t; *range = r; }
    }
}

// False where the layer's pieces are to be called one by one
static bool layer_plan(int S, int hidden, int Hq, int Hkv, int D, int mode, LayerPlan* q) {
    if (S <= 0 || Hq <= 0 || Hkv <= 0 || Hq % Hkv || D <= 0 || D % 4 || D > AL_MAXD || hidden <= 0 || hidden % 4 || S > 65535) return false;
    if ((long long)Hq * D > (1 << 17) || hidden > (1 << 17) || Hq > 65535) return false;
    LayerPlan& l = *q;
    l.collapsed = mode == BN_HEADS_COLLAPSED;
    if (l.collapsed && Hkv * D > AL_MAXW) return false;
    l.Wk = Hkv * D;
    l.Wq = l.collapsed ? l.Wk : Hq * D;
    l.W = l.collapsed ? l.Wk : D;
    l.problems = l.collapsed ? 1 : Hq;
    l.reps = l.collapsed ? 1 : Hq / Hkv;
    l.ld = l.Wq + 2 * l.Wk;
    project_plan(S, ceil_div(l.Wq, PJ_BN) + 2 * ceil_div(l.Wk, PJ_BN), hidden, &l.in_bm, &l.in_range);
    project_plan(S, ceil_div(hidden, PJ_BN), l.Wq, &l.out_bm, &l.out_range);
    // As many rows to a block as leave two blocks for every multiprocessor (rows share the reads of keys and values), and fit.
    const long long rows = (long long)S * l.problems, sms = sm_count();
    l.BM = l.wanted = rows >= 32 * sms ? 16 : rows >= 16 * sms ? 8 : rows >= 6 * sms ? 4 : rows > sms ? 2 : 1;
    l.p_ld = ceil_div(S, AL_KEYS) * AL_KEYS + 4;
    for (;; l.BM /= 2) {
        if (l.BM == 0) return false;
        l.smem = (size_t)(2 * AL_KEYS * (l.W + 16) + l.BM * (l.W + l.p_ld)) * sizeof(float);
        if (l.smem <= AL_SMEM) break;
    }
    size_t at = 0;
    auto take = [&](size_t floats) { const size_t was = at; at += (floats * sizeof(float) + 255) / 256 * 256; return was; };
    l.fold = l.collapsed && Hq > Hkv;
    l.wq_at = take(l.fold ? (size_t)hidden * l.Wq : 0);
    l.wo_at = take(l.fold ? (size_t)hidden * l.Wq : 0);
    l.part_at = take((size_t)ceil_div(hidden, l.in_range) * S * l.ld);
    l.rows_at = take((size_t)S * l.ld);
    l.attn_at = take((size_t)S * l.Wq);
    l.out_at = take(l.fold ? 0 : (size_t)ceil_div(l.Wq, l.out_range) * S * hidden);
    l.total = at;
    return true;
}

// Whether heads of their own go through tiles of 64 x 64, as a portion from the first position on
static bool layer_tiled(const LayerPlan& l, int S, int causal, int position_offset) { return !l.collapsed && causal && position_offset == 0 && S >= 64; }

// Whether the layer in one call is faster than its operators one by one.  It is, but for long sequences whose scores leave room for few
// rows to a block, and so read all keys and values for every one or two: relative times of a row and key here (the columns are read
// once for the BM rows) and in attn_f32_kernel (16 rows to a block, the scores over all query heads).  us as operators and in
// one call, collapsed and causal: 16 / 16 heads of 16, 7000 tokens (2 rows a block) 4905, 3911, 7900 tokens (1 row) 6028, 8430; 8 / 4 of
// 64, 15900 (1) 30500, 31793; 12 / 4 of 64, 15900 (1) 38417, 32037; 32 / 4 of 64, 8192 (1) 24193, 9537; 8 / 8 of 16, 16000 (2) 14091,
// 11066, 28000 (1) 42194, 62011; 4 / 4 of 16, 6000 (4) 1280, 840, 12000 (2) 3885, 4313; 8 / 2 of 32, 12000 (2) 6234, 4315, 30000 (1)
// 37041, 50612.  Per head, 4 / 2 of 64, not causal: 10000 (4) 22319, 16976, 13000 (2) 37317, 40138, 21000 (1) 97707, 195304.
static bool layer_best(const LayerPlan& l, int S, int Hq, int Hkv, int causal, int position_offset) {
    if (l.BM == l.wanted || layer_tiled(l, S, causal, position_offset)) return true;
    const float here = (0.8f + 0.0082f * l.W) / l.BM, apart = 0.25f + 0.0062f * l.W + (l.collapsed ? 0.003f * (Hq / Hkv - 1) * l.W : 0.f);
    return here <= apart;
}

template <int BM>
static int project_run(const ProjectParams& p, cudaStream_t st) {
    constexpr size_t smem = 2 * 3 * (BM * PJ_A_LD + PJ_KC * PJ_B_LD) * sizeof(__nv_bfloat16);
    if (int rc = allow_smem_once<project_kernel<BM>>(smem)) return rc;
    launch_dependent(project_kernel<BM>, dim3(p.tile_end[PJ_SETS - 1], ceil_div(p.M, BM), ceil_div(p.K, p.range)), BM * 4, smem, st, p);
    return launch_status("bn_attn_layer_f32");
}

static int project(int bm, ProjectParams p, cudaStream_t st) {
    for (int s = 0; s < PJ_SETS; ++s) p.tile_end[s] = (s ? p.tile_end[s - 1] : 0) + (s < p.sets ? ceil_div(p.set[s].N, PJ_BN) : 0);
    switch (bm) {
        case 32: return project_run<32>(p, st);
        case 64: return project_run<64>(p, st);
        default: return project_run<128>(p, st);
    }
}

template <int BM>
static int core_run(const LayerPlan& l, const CoreParams& p, cudaStream_t st) {
    if (int rc = allow_smem_once<attn_rows_f32_kernel<BM>>(l.smem)) return rc;
    launch_dependent(attn_rows_f32_kernel<BM>, dim3(ceil_div(p.S, BM), p.problems), AL_THREADS, l.smem, st, p);
    return launch_status("bn_attn_layer_f32");
}

static int core(const LayerPlan& l, const CoreParams& p, cudaStream_t st) {
    if (l.tiled) {                                             // heads of their own: as a portion from the first position on
        AttnPortionParams t{};
        t.q = p.rows; t.k = p.rows + p.k_at; t.v = p.rows + p.v_at; t.out = p.out;
        t.q_ld = t.k_ld = t.v_ld = p.ld; t.out_ld = (int64_t)p.problems * p.W;
        t.k_head = t.v_head = p.W;
        t.B = 1; t.S = t.rows_per_seq = p.S; t.H = p.problems; t.kv_heads = p.problems / p.reps; t.dim = t.vdim = p.W;
        t.mask = MASK_CHUNK; t.span = 1 << 30; t.scale = p.scale;
        return attn_any(t, 0, st, "bn_attn_layer_f32");
    }
    switch (l.BM) {
        case 1: return core_run<1>(l, p, st);
        case 2: return core_run<2>(l, p, st);
        case 4: return core_run<4>(l, p, st);
        case 8: return core_run<8>(l, p, st);
        default: return core_run<16>(l, p, st);
    }
}

template <int WARPS>
static int out_run(const OutParams& p, cudaStream_t st) {
    const size_t smem = (size_t)3 * ceil_div(p.W, 16) * 16 * OUT_LD * sizeof(__nv_bfloat16);
    if (int rc = allow_smem_once<out_kernel<WARPS>>(smem)) return rc;
    launch_dependent(out_kernel<WARPS>, dim3(ceil_div(p.hidden, OUT_BN), ceil_div(p.S, 16 * WARPS)), WARPS * 32, smem, st, p);
    return launch_status("bn_attn_layer_f32");
}

}  // namespace bn

using namespace bn;

extern "C" size_t bn_attn_layer_f32_workspace_bytes(int S, int hidden, int Hq, int Hkv, int D, int heads_mode) {
    LayerPlan l;
    return (heads_mode == BN_HEADS_COLLAPSED || heads_mode == BN_HEADS_PER_HEAD) && layer_plan(S, hidden, Hq, Hkv, D, heads_mode, &l) ? l.total : 0;
}

extern "C" size_t bn_attn_layer_f32_best_bytes(int S, int hidden, int Hq, int Hkv, int D, int position_offset, int causal, int heads_mode) {
    LayerPlan l;
    return (heads_mode == BN_HEADS_COLLAPSED || heads_mode == BN_HEADS_PER_HEAD) && layer_plan(S, hidden, Hq, Hkv, D, heads_mode, &l) &&
           layer_best(l, S, Hq, Hkv, causal, position_offset) ? l.total : 0;
}

extern "C" int bn_attn_layer_f32(const float* x, int64_t x_rs, const float* wq, int64_t wq_rs, const float* wk, int64_t wk_rs,
                                 const float* wv, int64_t wv_rs, const float* wo, int64_t wo_rs, float* out, int64_t out_rs, int S,
                                 int hidden, int Hq, int Hkv, int D, float scale, float theta, int position_offset, int causal,
                                 int heads_mode, void* workspace, size_t workspace_bytes, bn_stream_t stream) {
    const char* what = "bn_attn_layer_f32";
    if (!x || !wq || !wk || !wv || !wo || !out || !workspace) return fail(BN_ERR_INVALID_ARG, "%s: null pointer", what);
    if (heads_mode != BN_HEADS_COLLAPSED && heads_mode != BN_HEADS_PER_HEAD) return fail(BN_ERR_INVALID_ARG, "%s: heads_mode=%d", what, heads_mode);
    LayerPlan l;
    if (!layer_plan(S, hidden, Hq, Hkv, D, heads_mode, &l)) return fail(BN_ERR_UNSUPPORTED, "%s: S=%d hidden=%d Hq=%d Hkv=%d D=%d", what, S, hidden, Hq, Hkv, D);
    uintptr_t bits = 0;
    for (const void* a : {(const void*)x, (const void*)wq, (const void*)wk, (const void*)wv, (const void*)wo, (const void*)out, (const void*)workspace})
        bits |= reinterpret_cast<uintptr_t>(a);
    if ((bits & 15) || ((x_rs | wq_rs | wk_rs | wv_rs | wo_rs | out_rs) & 3))
        return fail(BN_ERR_INVALID_ARG, "%s: operands must be 16-byte aligned rows", what);
    if (workspace_bytes < l.total) return fail(BN_ERR_WORKSPACE, "%s: %zu bytes of scratch, %zu needed", what, workspace_bytes, l.total);
    if (int rc = require_sm100()) return rc;
    cudaStream_t st = as_stream(stream);
    char* ws = static_cast<char*>(workspace);
    auto at = [&](size_t offset) { return reinterpret_cast<float*>(ws + offset); };
    const int reps = Hq / Hkv, most = 8 * sm_count();
    if (l.fold) {
        const long long blocks = ((long long)hidden * l.Wq / 4 + AL_THREADS - 1) / AL_THREADS;
        launch_dependent(fold_kernel, dim3((unsigned)(blocks < most ? blocks : most)), AL_THREADS, 0, st, wq, wq_rs, at(l.wq_at), hidden, Hkv, reps, D);
        if (int rc = launch_status(what)) return rc;
    }
    const ProjectParams in{x, x_rs, at(l.part_at), S, hidden, l.ld, l.in_range, 3,
                           {{l.fold ? at(l.wq_at) : wq, l.fold ? l.Wq : wq_rs, l.Wq}, {wk, wk_rs, l.Wk}, {wv, wv_rs, l.Wk}}, {}};
    if (int rc = project(l.in_bm, in, st)) return rc;
    const FinishParams fin{at(l.part_at), at(l.rows_at), ceil_div(hidden, l.in_range), S, l.Wq, l.Wk, D, position_offset, theta,
                           wo, at(l.wo_at), wo_rs, hidden, reps};
    launch_dependent(finish_kernel, dim3(S + (l.fold ? 4 * sm_count() : 0)), AL_THREADS, 0, st, fin);
    if (int rc = launch_status(what)) return rc;
    const CoreParams c{at(l.rows_at), at(l.attn_at), S, l.ld, l.Wq, l.Wq + l.Wk, l.W, l.problems, l.reps, l.p_ld, scale, position_offset, causal};
    l.tiled = layer_tiled(l, S, causal, position_offset);
    if (int rc = core(l, c, st)) return rc;
    if (l.collapsed && (l.fold || wo_rs == hidden)) {
        const OutParams o{at(l.attn_at), l.fold ? at(l.wo_at) : wo, out, out_rs, S, l.W, hidden};
        return S > 64 ? out_run<8>(o, st) : out_run<4>(o, st);
    }
    const ProjectParams o{at(l.attn_at), l.Wq, at(l.out_at), S, l.Wq, hidden, l.out_range, 1, {{wo, wo_rs, hidden}}, {}};
    if (int rc2 = project(l.out_bm, o, st)) return rc2;
    const long long blocks = ((long long)S * hidden / 4 + AL_THREADS - 1) / AL_THREADS;
    launch_dependent(add_ranges_kernel, dim3((unsigned)(blocks < most ? blocks : most)), AL_THREADS, 0, st, (const float*)at(l.out_at), out,
                     out_rs, S, hidden, ceil_div(l.Wq, l.out_range));
    return launch_status(what);
}
