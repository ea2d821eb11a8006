// The fp32 attention layer in one call: q, k, v projections, RoPE, causal softmax attention (collapsed heads or one softmax per
// query head) and the output projection (reference sequence: mygrad/llama/llama_layers.py:155-186).
//
// Collapsed heads have ONE softmax over the scores summed over all query heads.  The reps query heads that share a key head meet
// the same keys, at the same rotation, so  sum_h rot(q_h) . rot(k) = rot(sum_h q_h) . rot(k),  and a sum of heads is a product
// with the sum of their weight columns; the reps output heads are one and the same, so the output projection reads them with the
// sum of its weight rows.  32 query heads over 4 key heads of 64: 2048 columns of q, of every score and of the output
// projection's K become 256.  The kernels that stream the weights sum them on the way (reading them is what the layer cannot do
// without); every sum is fp32, and shorter than the one it replaces.
//
// 128 rows, width 2048, 32 / 4 heads of 64, collapsed: 47 us; as four operators (three products in a launch, scores of 2048 columns,
// output projection of K = 2048) 215 us.  Error against 64 bits (2-norm) 8e-7, before 3.8e-6.  Per head 114 us, before 158 us.
//
//   1 project_kernel    x @ [Wq | Wk | Wv] over ranges of k           3 attn_rows_f32_kernel   softmax attention
//   2 finish_kernel     the ranges added up, q and k rotated          4 out_kernel (collapsed), or project_kernel + add_ranges_kernel
#include "common.cuh"
#include "hybrid.cuh"
#include "ptx.cuh"

namespace bn {

constexpr int AL_THREADS = 256, AL_MAXW = 256, AL_MAXD = 64;
constexpr size_t AL_SMEM = 200 * 1024;

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

// ---- 1: C[z] = A[:, range z] @ B[range z, :], FMA chains with k ascending.
// A block has 32 TM rows, 64 columns and a range of k, which it walks in chunks of 32 through three stages of shared memory: A, and a
// B whose columns stand for themselves, by cp.async; the columns of a B that are sums of heads are loaded into registers while a
// chunk is multiplied, and summed and stored behind it.  512 threads of TM x 4 outputs, rows 32 apart; what bounds a block is reading
// shared memory (8 16-byte reads of 4 cycles for 64 FMAs at TM = 4).  128 rows, collapsed (2048 -> 256 + 256 + 256): 18 us.
constexpr int PJ_BN = 64, PJ_KC = 32, PJ_STAGES = 3, PJ_SETS = 3, PJ_THREADS = 512;
struct ProjectSet {
    const float* B;
    int64_t b_rs;
    int N, reps, D;              // N columns, each the sum of `reps` columns, heads of D
};
struct ProjectParams {
    const float* A;
    int64_t a_rs;
    float* C;                    // [ranges][M][ld]
    int M, K, ld, range, sets;
    ProjectSet set[PJ_SETS];
    int tile_end[PJ_SETS];
};

template <int TM>
__global__ void __launch_bounds__(PJ_THREADS) project_kernel(const __grid_constant__ ProjectParams p) {
    constexpr int BM = 32 * TM, A_LD = PJ_KC + 4, A_STAGE = BM * A_LD, B_STAGE = PJ_KC * PJ_BN;
    extern __shared__ __align__(16) float al_smem[];
    const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16, tile = blockIdx.x;
    const int s = (tile >= p.tile_end[0]) + (tile >= p.tile_end[1]);
    const ProjectSet& q = p.set[s];
    const int tile0 = s ? p.tile_end[s - 1] : 0, col = (tile - tile0) * PJ_BN + tx * 4, row0 = blockIdx.y * BM;
    const int k0 = blockIdx.z * p.range, kn = min(p.K - k0, p.range), chunks = (kn + PJ_KC - 1) / PJ_KC;
    float* As = al_smem;                                       // [stage][BM][36]
    float* Bs = As + PJ_STAGES * A_STAGE;                      // [stage][32][64]
    const uint32_t uA = ptx::smem_u32(As), uB = ptx::smem_u32(Bs);
    const bool col_in = col < q.N, sums = q.reps > 1;
    const float* b_col = q.B + (col_in ? sums ? (int64_t)(col / q.D) * q.reps * q.D + col % q.D : col : 0);
    ptx::grid_dependency_wait();
    ptx::grid_launch_dependents();
    float4 heads[8];
    // this thread's four columns of row ty of chunk c: the first eight heads
    auto ask_heads = [&](int c) {
        const int k = c * PJ_KC + ty;
        const float* at = b_col + (int64_t)(k0 + k) * q.b_rs;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            heads[i] = k < kn && col_in && i < q.reps ? __ldcg(reinterpret_cast<const float4*>(at + i * q.D)) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    auto put_heads = [&](int c) {
        float4 v = add4(add4(add4(heads[0], heads[1]), add4(heads[2], heads[3])), add4(add4(heads[4], heads[5]), add4(heads[6], heads[7])));
        const int k = c * PJ_KC + ty;
        if (q.reps > 8 && k < kn && col_in) v = add4(v, sum_heads(b_col + (int64_t)(k0 + k) * q.b_rs + 8 * q.D, q.D, q.reps - 8));
        *reinterpret_cast<float4*>(Bs + (c % PJ_STAGES) * B_STAGE + ty * PJ_BN + tx * 4) = v;
    };
    // K and the range are multiples of 4, so a piece of four k lies inside or outside; what lies outside becomes zero
    auto ask = [&](int c) {
        if (c < chunks) {
            const int st = c % PJ_STAGES, kc = c * PJ_KC;
#pragma unroll
            for (int e = tid; e < BM * (PJ_KC / 4); e += PJ_THREADS) {
                const int r = e / (PJ_KC / 4), k = e % (PJ_KC / 4) * 4;
                const bool in = row0 + r < p.M && kc + k < kn;
                ptx::cp_async_16(uA + (st * A_STAGE + r * A_LD + k) * 4, in ? p.A + (row0 + r) * p.a_rs + k0 + kc + k : p.A, in ? 16 : 0);
            }
            if (!sums) {
                const bool in = col_in && kc + ty < kn;
                ptx::cp_async_16(uB + (st * B_STAGE + ty * PJ_BN + tx * 4) * 4, in ? b_col + (int64_t)(k0 + kc + ty) * q.b_rs : q.B, in ? 16 : 0);
            }
        }
        ptx::cp_async_commit();
    };
    ask(0);
    ask(1);
    if (sums)
        for (int c = 0; c < 2 && c < chunks; ++c) {
            ask_heads(c);
            put_heads(c);
        }
    float acc[TM][4];
#pragma unroll
    for (int i = 0; i < TM; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    for (int c = 0; c < chunks; ++c) {
        ptx::cp_async_wait<1>();
        __syncthreads();                                       // chunk c is there, and chunk c - 1, whose stage c + 2 takes, has been read
        ask(c + 2);
        if (sums && c + 2 < chunks) ask_heads(c + 2);
        const float* a = As + (c % PJ_STAGES) * A_STAGE + ty * A_LD;
        const float* b = Bs + (c % PJ_STAGES) * B_STAGE + tx * 4;
#pragma unroll
        for (int k = 0; k < PJ_KC; k += 4) {
            float4 av[TM], bv[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) bv[e] = *reinterpret_cast<const float4*>(b + (k + e) * PJ_BN);
#pragma unroll
            for (int i = 0; i < TM; ++i) av[i] = *reinterpret_cast<const float4*>(a + i * 32 * A_LD + k);
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    const float x = e == 0 ? av[i].x : e == 1 ? av[i].y : e == 2 ? av[i].z : av[i].w;
                    acc[i][0] = fmaf(x, bv[e].x, acc[i][0]);
                    acc[i][1] = fmaf(x, bv[e].y, acc[i][1]);
                    acc[i][2] = fmaf(x, bv[e].z, acc[i][2]);
                    acc[i][3] = fmaf(x, bv[e].w, acc[i][3]);
                }
        }
        if (sums && c + 2 < chunks) put_heads(c + 2);
    }
    if (!col_in) return;
    int at = col;                                              // the sets' columns lie side by side
    for (int i = 0; i < s; ++i) at += p.set[i].N;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int r = row0 + ty + i * 32;
        if (r < p.M)
            *reinterpret_cast<float4*>(p.C + ((int64_t)blockIdx.z * p.M + r) * p.ld + at) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    }
}

// ---- 2
struct FinishParams {
    const float* part;           // [ranges][S][Wq + 2 Wk]
    float* rows;                 // [S][Wq + 2 Wk]: rotated q | rotated k | v
    int ranges, S, Wq, Wk, D, offset;
    float theta;
};

// A block per row: the angles of its position are worked out once.
__global__ void __launch_bounds__(AL_THREADS) finish_kernel(const FinishParams p) {
    __shared__ float2 turn[AL_MAXD / 2];
    const int tid = threadIdx.x, half = p.D / 2, ld = p.Wq + 2 * p.Wk;
    const int row = blockIdx.x;
    if (tid < half) {
        const float angle = (row + p.offset) * rope_inv_freq(tid, p.D, p.theta);
        float cos_angle, sin_angle;
        sincosf(angle, &sin_angle, &cos_angle);
        turn[tid] = make_float2(cos_angle, sin_angle);
    }
    __syncthreads();
    ptx::grid_dependency_wait();
    ptx::grid_launch_dependents();
    const int64_t range = (int64_t)p.S * ld;
    for (int c = tid * 4; c < ld; c += AL_THREADS * 4) {
        const float* at = p.part + (int64_t)row * ld + c;
        float4 s = *reinterpret_cast<const float4*>(at);
#pragma unroll 4
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
// head: W = D); tiles of KEYS keys by cp.async, two in flight (32 keys where W is wide, so that the next kernel's blocks find room
// beside).  256 / KEYS threads share a key, each takes its groups of four columns in turn for all BM rows (with the row stride of
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

template <int BM, int KEYS>
__global__ void __launch_bounds__(AL_THREADS) attn_rows_f32_kernel(const CoreParams p) {
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
    auto ask_keys = [&](int t) {
        if (t < tiles)
            for (int e = tid; e < KEYS * quads; e += AL_THREADS) {
                const int r = e / quads, c = e % quads * 4;
                const bool in = t * KEYS + r < p.S;
                ptx::cp_async_16(uK + (((t & 1) * KEYS + r) * k_ld + c) * 4, k + (in ? (int64_t)(t * KEYS + r) * p.ld + c : 0), in ? 16 : 0);
            }
        ptx::cp_async_commit();
    };
    for (int e = tid; e < BM * quads; e += AL_THREADS) {
        const int r = e / quads, c = e % quads * 4;
        const bool in = row0 + r < p.S;
        ptx::cp_async_16(uQ + (r * W + c) * 4, q + (in ? (int64_t)(row0 + r) * p.ld + c : 0), in ? 16 : 0);
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
    const int parts = AL_THREADS / quads, c4 = tid % quads, vp = tid / quads;
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
        const float* vc = v + c4 * 4;
        int j = vp;
        const int all = row0 + BM <= p.S ? row_last(0) : -1;   // keys up to here are seen by all the rows
#pragma unroll(BM <= 2 ? 16 : 8)
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

// ---- 4 (collapsed): out = attn (S, W) @ the sums of wo's rows over the heads of a group.  A block has 64 TM rows and 16
// columns; it sums its part of the weight before it waits for the attention (`wo` is as old as the call: the first launch of the
// call has waited for what wrote it), so that behind the attention come one round trip for its rows and W FMAs a thread and output.
constexpr int OUT_BN = 16, OUT_THREADS = 256;
struct OutParams {
    const float* attn;           // [S][W]
    const float* wo;             // [W / D * reps * D][hidden]
    float* out;
    int64_t wo_rs, out_rs;
    int S, W, D, reps, hidden;
};

template <int TM>
__global__ void __launch_bounds__(OUT_THREADS) out_kernel(const OutParams p) {
    constexpr int BM = 64 * TM;
    extern __shared__ __align__(16) float al_smem[];
    const int tid = threadIdx.x, tx = tid % 4, ty = tid / 4, row0 = blockIdx.y * BM, col = blockIdx.x * OUT_BN + tx * 4, a_ld = p.W + 4;
    float* Bs = al_smem;                                       // [W][16]
    float* As = Bs + p.W * OUT_BN;                             // [BM][W + 4]
    const bool col_in = col < p.hidden;
#pragma unroll 2
    for (int k = ty; k < p.W; k += 64)
        *reinterpret_cast<float4*>(Bs + k * OUT_BN + tx * 4) =
            col_in ? sum_heads(p.wo + ((int64_t)(k / p.D) * p.reps * p.D + k % p.D) * p.wo_rs + col, (int64_t)p.D * p.wo_rs, p.reps)
                   : make_float4(0.f, 0.f, 0.f, 0.f);
    ptx::grid_dependency_wait();
    ptx::grid_launch_dependents();
    const uint32_t uA = ptx::smem_u32(As);
    const int quads = p.W / 4, lane = tid % 32;
    for (int r = tid / 32; r < BM; r += OUT_THREADS / 32) {
        const bool in = row0 + r < p.S;
        const float* at = p.attn + (in ? (int64_t)(row0 + r) * p.W : 0);
        for (int c = lane; c < quads; c += 32) ptx::cp_async_16(uA + (r * a_ld + c * 4) * 4, at + c * 4, in ? 16 : 0);
    }
    ptx::cp_async_wait_all();
    __syncthreads();
    float acc[TM][4];
#pragma unroll
    for (int i = 0; i < TM; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    const float* a = As + ty * a_ld;
    const float* b = Bs + tx * 4;
#pragma unroll 4
    for (int k = 0; k < p.W; k += 4) {
        float4 av[TM], bv[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) bv[e] = *reinterpret_cast<const float4*>(b + (k + e) * OUT_BN);
#pragma unroll
        for (int i = 0; i < TM; ++i) av[i] = *reinterpret_cast<const float4*>(a + i * 64 * a_ld + k);
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const float x = e == 0 ? av[i].x : e == 1 ? av[i].y : e == 2 ? av[i].z : av[i].w;
                acc[i][0] = fmaf(x, bv[e].x, acc[i][0]);
                acc[i][1] = fmaf(x, bv[e].y, acc[i][1]);
                acc[i][2] = fmaf(x, bv[e].z, acc[i][2]);
                acc[i][3] = fmaf(x, bv[e].w, acc[i][3]);
            }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int r = row0 + ty + i * 64;
        if (col_in && r < p.S) *reinterpret_cast<float4*>(p.out + r * p.out_rs + col) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    }
}

// Lets `kernel` have so much shared memory; asked of the driver once per thread and device for each kernel (`known`)
struct SmemKnown {
    int dev = -1;
    size_t bytes = 0;
};
template <typename K>
static int allow_smem_once(K kernel, size_t bytes, SmemKnown& known) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev == known.dev && bytes <= known.bytes) return BN_OK;
    if (int rc = allow_smem(kernel, bytes, "bn_attn_layer_f32")) return rc;
    known.dev = dev;
    known.bytes = bytes;
    return BN_OK;
}

struct LayerPlan {
    int Wq, Wk, W, problems, reps, ld, in_tm, in_range, out_tm, out_range, BM, keys, p_ld;
    bool collapsed;
    size_t part_at, rows_at, attn_at, out_at, total, smem;
};

// Rows to a block, and how K is cut: whole rounds of blocks, two to a multiprocessor, each of which takes about 2 us and 8 ns a k and
// 32 rows of its block, half of that while it is alone there.  A range is a write and a read of the result more.
static void project_plan(int M, int tiles, int K, int* tm, int* range) {
    const int sms = sm_count();
    *tm = M > 64 ? 4 : M > 32 ? 2 : 1;
    const long long blocks = (long long)tiles * ceil_div(M, 32 * *tm);
    float least = 1e30f;
    for (int n = 1; n <= 32 && (n == 1 || K / n >= PJ_KC); ++n) {
        const int r = ceil_div(ceil_div(K, n), PJ_KC) * PJ_KC, ranges = ceil_div(K, r);
        const long long busy = (blocks * ranges + sms - 1) / sms;          // blocks that the busiest multiprocessor has
        const float t = 2.f * ((busy + 1) / 2) + busy * r * 8e-3f * *tm + 2.5e-6f * M * tiles * PJ_BN * ranges / 4;
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
    project_plan(S, ceil_div(l.Wq, PJ_BN) + 2 * ceil_div(l.Wk, PJ_BN), hidden, &l.in_tm, &l.in_range);
    project_plan(S, ceil_div(hidden, PJ_BN), l.Wq, &l.out_tm, &l.out_range);
    // As many rows to a block as leave two blocks for every multiprocessor (rows share the reads of keys and values), and fit.
    const long long rows = (long long)S * l.problems, sms = sm_count();
    l.BM = rows >= 32 * sms ? 16 : rows >= 16 * sms ? 8 : rows >= 6 * sms ? 4 : rows > sms ? 2 : 1;
    l.keys = l.W > 128 ? 32 : 64;
    l.p_ld = ceil_div(S, l.keys) * l.keys + 4;
    for (;; l.BM /= 2) {
        if (l.BM == 0) return false;
        l.smem = (size_t)(2 * l.keys * (l.W + 16) + l.BM * (l.W + l.p_ld)) * sizeof(float);
        if (l.smem <= AL_SMEM) break;
    }
    size_t at = 0;
    auto take = [&](size_t floats) { const size_t was = at; at += (floats * sizeof(float) + 255) / 256 * 256; return was; };
    l.part_at = take((size_t)ceil_div(hidden, l.in_range) * S * l.ld);
    l.rows_at = take((size_t)S * l.ld);
    l.attn_at = take((size_t)S * l.Wq);
    l.out_at = take(l.collapsed ? 0 : (size_t)ceil_div(l.Wq, l.out_range) * S * hidden);
    l.total = at;
    return true;
}

template <int TM>
static int project_run(const ProjectParams& p, cudaStream_t st) {
    static thread_local SmemKnown known;
    const size_t smem = (size_t)PJ_STAGES * (32 * TM * (PJ_KC + 4) + PJ_KC * PJ_BN) * sizeof(float);
    if (int rc = allow_smem_once(project_kernel<TM>, smem, known)) return rc;
    launch_dependent(project_kernel<TM>, dim3(p.tile_end[PJ_SETS - 1], ceil_div(p.M, 32 * TM), ceil_div(p.K, p.range)), PJ_THREADS, smem, st, p);
    return launch_status("bn_attn_layer_f32");
}

static int project(int tm, ProjectParams p, cudaStream_t st) {
    for (int s = 0; s < PJ_SETS; ++s) p.tile_end[s] = (s ? p.tile_end[s - 1] : 0) + (s < p.sets ? ceil_div(p.set[s].N, PJ_BN) : 0);
    switch (tm) {
        case 1: return project_run<1>(p, st);
        case 2: return project_run<2>(p, st);
        default: return project_run<4>(p, st);
    }
}

template <int BM, int KEYS>
static int core_run(const LayerPlan& l, const CoreParams& p, cudaStream_t st) {
    static thread_local SmemKnown known;
    if (int rc = allow_smem_once(attn_rows_f32_kernel<BM, KEYS>, l.smem, known)) return rc;
    launch_dependent(attn_rows_f32_kernel<BM, KEYS>, dim3(ceil_div(p.S, BM), p.problems), AL_THREADS, l.smem, st, p);
    return launch_status("bn_attn_layer_f32");
}

template <int KEYS>
static int core(const LayerPlan& l, const CoreParams& p, cudaStream_t st) {
    switch (l.BM) {
        case 1: return core_run<1, KEYS>(l, p, st);
        case 2: return core_run<2, KEYS>(l, p, st);
        case 4: return core_run<4, KEYS>(l, p, st);
        case 8: return core_run<8, KEYS>(l, p, st);
        default: return core_run<16, KEYS>(l, p, st);
    }
}

template <int TM>
static int out_run(const OutParams& p, cudaStream_t st) {
    static thread_local SmemKnown known;
    const size_t smem = (size_t)(p.W * OUT_BN + 64 * TM * (p.W + 4)) * sizeof(float);
    if (int rc = allow_smem_once(out_kernel<TM>, smem, known)) return rc;
    launch_dependent(out_kernel<TM>, dim3(ceil_div(p.hidden, OUT_BN), ceil_div(p.S, 64 * TM)), OUT_THREADS, smem, st, p);
    return launch_status("bn_attn_layer_f32");
}

}  // namespace bn

using namespace bn;

extern "C" size_t bn_attn_layer_f32_workspace_bytes(int S, int hidden, int Hq, int Hkv, int D, int heads_mode) {
    LayerPlan l;
    return (heads_mode == BN_HEADS_COLLAPSED || heads_mode == BN_HEADS_PER_HEAD) && layer_plan(S, hidden, Hq, Hkv, D, heads_mode, &l) ? l.total : 0;
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
    const int reps = Hq / Hkv;
    const ProjectParams in{x, x_rs, at(l.part_at), S, hidden, l.ld, l.in_range, 3,
                           {{wq, wq_rs, l.Wq, l.collapsed ? reps : 1, D}, {wk, wk_rs, l.Wk, 1, D}, {wv, wv_rs, l.Wk, 1, D}}, {}};
    if (int rc = project(l.in_tm, in, st)) return rc;
    const FinishParams fin{at(l.part_at), at(l.rows_at), ceil_div(hidden, l.in_range), S, l.Wq, l.Wk, D, position_offset, theta};
    launch_dependent(finish_kernel, dim3(S), AL_THREADS, 0, st, fin);
    if (int rc = launch_status(what)) return rc;
    const CoreParams c{at(l.rows_at), at(l.attn_at), S, l.ld, l.Wq, l.Wq + l.Wk, l.W, l.problems, l.reps, l.p_ld, scale, position_offset, causal};
    if (int rc = l.keys == 32 ? core<32>(l, c, st) : core<64>(l, c, st)) return rc;
    if (l.collapsed) {
        const OutParams o{at(l.attn_at), wo, out, wo_rs, out_rs, S, l.W, D, reps, hidden};
        return S > 64 ? out_run<2>(o, st) : out_run<1>(o, st);
    }
    const ProjectParams o{at(l.attn_at), l.Wq, at(l.out_at), S, l.Wq, hidden, l.out_range, 1, {{wo, wo_rs, hidden, 1, D}}, {}};
    if (int rc2 = project(l.out_tm, o, st)) return rc2;
    const long long blocks = ((long long)S * hidden / 4 + AL_THREADS - 1) / AL_THREADS, most = 8 * sm_count();
    launch_dependent(add_ranges_kernel, dim3((unsigned)(blocks < most ? blocks : most)), AL_THREADS, 0, st, (const float*)at(l.out_at), out,
                     out_rs, S, hidden, ceil_div(l.Wq, l.out_range));
    return launch_status(what);
}
