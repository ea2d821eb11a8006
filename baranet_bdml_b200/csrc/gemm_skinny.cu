// C (M,N) bf16 = A (M,K) bf16 @ Bt (N,K)^T bf16 for M <= 16 rows: the projections of a decode step, where every
// sequence contributes ONE row (mygrad/llama/llama_layers.py:157-159,186 and the MLP, :217-232, applied to the new
// token only; reference operator op_mm, src/ops/op_mm.cuh:39-57, whose naive kernel runs for such shapes).
//
// With so few rows the product is a stream of the weight matrix through the SMs: 2 FLOP per weight byte and row, far
// below what the tensor cores need, so the bound is HBM bandwidth and what matters is that every SM has many loads in
// flight.  The 128-row tcgen05 tiles of the large GEMM are the wrong tool here (an eighth of each instruction would do
// useful work and a tile's ring holds few bytes in flight); this kernel uses warp-level mma.sync.m16n8k16, whose M = 16
// is the whole batch:
//   CTA = 8 warps = 8 output columns (8 rows of Bt); warp w takes the w-th eighth of K for all 8 columns.
//   A lane loads 16 contiguous bytes (8 bf16 along K) of ONE weight row and of two activation rows per 32-wide K step
//   (in batches of 4 or 8 steps, weight and activation loads of a batch all in flight before the first use).  The K order inside a step
//   is whatever this lane assignment gives: a dot product does not care, as long as A and B use the same one, so no
//   shuffles or shared-memory staging are needed to form the MMA fragments.
//   The 8 warps' partial sums (16 x 8 fp32) are added through shared memory in warp order (deterministic).
// Variants: up to three column ranges of one concatenated weight written to separate outputs (q, k, v of the layer in one
// launch); the same with the K and V ranges rotated / appended to the paged cache by the epilogue instead (what
// bn_kv_append would do with them, mygrad/llama/llama_layers.py:161-171 for the new token); and the gated pair (two weights, h = act(x Wg) * (x Wu); SwiGLU: op_silu.cuh:7-15);
// an fp32 output; the result's activation times a matrix given by the caller; and the activation of the result plus a bias.
// Most products with a K that is a multiple of 256 take the second kernel of this file, whose CTAs stay (gemm_wide_kernel).
// K is a multiple of 8 and at most 8192, N a multiple of 8.  When K is a multiple of 256 a warp's eighth is a whole number
// of 32-wide steps; otherwise (RAGGED) the eighths are rounded up and pieces beyond K read as zero.  Anything else belongs to bn_gemm_bf16_nt_small_m.
#include "common.cuh"
#include "hybrid.cuh"
#include "ptx.cuh"

namespace bn {

using namespace ptx;

constexpr int SK_WARPS = 8;
constexpr int SK_MAX_STEPS = 32;        // 32-wide K steps per warp: K <= 8 * 32 * 32 = 8192

struct SkinnyParams {
    const __nv_bfloat16* a;             // (M, K)
    const __nv_bfloat16* bt;            // (N, K)
    const __nv_bfloat16* bt2;           // SwiGLU: the up weight (N, K); bt is the gate weight
    __nv_bfloat16* out[3];              // outputs of the column ranges
    int n_end[3];                       // range r covers columns [n_end[r-1], n_end[r])
    int ld[3];                          // row stride of out[r] in elements
    int M, N, K, steps;                 // steps = K / (8 * 32), rounded up
    float* out32;                       // when set, the (single) output range in fp32 instead of out[0]
    bool rounded;                       // ... of the sum rounded to bf16
    const __nv_bfloat16* mul;           // when set, out[0] = act(x W) * mul, mul (M, mul_ld)
    long long mul_ld;
    int act;                            // of the gated pair, of `mul`, or of the result plus bias
    const float* bias;                  // optional, (N)
    // APPEND: columns from n_end[0] on are the K and V projections of one new token per row and go to the paged cache
    // instead of out[1] / out[2] (arguments as bn_kv_append)
    __nv_bfloat16* pool;
    const int32_t* page_table;
    const int32_t* seq_ids;
    const int32_t* positions;
    int64_t pool_pages;
    int max_pages, Hkv, D;
    float theta;
};

// Where a finished sum of row `row`, column n goes, and what is done to it on the way
template <bool GLU>
__device__ __forceinline__ void skinny_store(const SkinnyParams& p, int row, int n, float v) {
    if (p.out32) {
        p.out32[(size_t)row * p.N + n] = p.rounded ? __bfloat162float(__float2bfloat16(v)) : v;
        return;
    }
    if (p.bias) v += __ldg(p.bias + n);
    if (!GLU) v = activation_fast(p.act, v);
    if (p.mul) v *= __bfloat162float(p.mul[row * p.mul_ld + n]);
    // selects, not indexed parameter arrays (an index known only at run time would copy them to local memory)
    __nv_bfloat16* o = p.out[0];
    int ld = p.ld[0], first = 0;
    if (n >= p.n_end[1]) { o = p.out[2]; ld = p.ld[2]; first = p.n_end[1]; }
    else if (n >= p.n_end[0]) { o = p.out[1]; ld = p.ld[1]; first = p.n_end[0]; }
    o[(size_t)row * ld + (n - first)] = __float2bfloat16(v);
}

// APPEND: what bn_kv_append does with the bf16 row the plain kernel would have written: the value is rounded to bf16 first, a K pair
// (2i, 2i+1) = (this column, its neighbour's lane) is rotated at the row's position in fp32 and rounded again, V is stored as it
// is - the cache ends up with the bits of the two-launch path.  Whole warps call it.
__device__ __forceinline__ void skinny_append(const SkinnyParams& p, int row, int n, float v) {
    const float vb = __bfloat162float(__float2bfloat16(v));
    const float other = __shfl_xor_sync(0xffffffffu, vb, 1);
    if (row < p.M) {
        const bool is_k = n < p.n_end[1];
        const int local = n - (is_k ? p.n_end[0] : p.n_end[1]);
        const int g = local / p.D, d = local - g * p.D;
        const int pos = p.positions[row];
        const int lp = pos / BN_PAGE_TOKENS;
        if (pos >= 0 && lp < p.max_pages) {
            const int page = p.page_table[(int64_t)p.seq_ids[row] * p.max_pages + lp];
            if (page >= 0 && page < p.pool_pages) {
                float y = vb;
                if (is_k) {
                    const float angle = pos * rope_inv_freq(d / 2, p.D, p.theta);
                    const float c = cosf(angle), sn = sinf(angle);
                    y = (d & 1) ? other * sn + vb * c : vb * c - other * sn;
                }
                p.pool[((((int64_t)page * p.Hkv + g) * 2 + (is_k ? 0 : 1)) * BN_PAGE_TOKENS + pos % BN_PAGE_TOKENS) * p.D + d] =
                    __float2bfloat16(y);
            }
        }
    }
}

// CH = K steps whose loads a lane keeps in flight at once.  More of them cover more latency per warp; fewer leave
// registers for more CTAs per SM (8: two, 2: four), which matters when the grid would otherwise need a second, nearly
// empty wave.
template <bool SWIGLU, int CH, bool APPEND = false, bool RAGGED = false>
__global__ void __launch_bounds__(SK_WARPS * 32, CH == 8 ? 2 : SWIGLU ? 3 : 4)
gemm_skinny_kernel(const SkinnyParams p) {
    __shared__ float s_part[SK_WARPS][2][16][8 + 1];
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int g = lane / 4, j = lane % 4;                 // weight row inside the CTA's 8 / which 8 of a step's 32 K positions
    const int n0 = blockIdx.x * 8;
    const size_t kbase = (size_t)warp * p.steps * 32 + j * 8;
    const uint4* bw = reinterpret_cast<const uint4*>(p.bt + (size_t)(n0 + g) * p.K + kbase);
    const uint4* bw2 = SWIGLU ? reinterpret_cast<const uint4*>(p.bt2 + (size_t)(n0 + g) * p.K + kbase) : nullptr;
    const uint4* a_lo = reinterpret_cast<const uint4*>(p.a + (size_t)g * p.K + kbase);
    const uint4* a_hi = reinterpret_cast<const uint4*>(p.a + (size_t)(g + 8) * p.K + kbase);
    const bool lo_ok = g < p.M, hi_ok = g + 8 < p.M;
    float acc[4] = {0.f, 0.f, 0.f, 0.f}, acc2[4] = {0.f, 0.f, 0.f, 0.f};
    // Loads first, arithmetic after: for a batch of K steps the lane requests its pieces of the weight rows (evict-first:
    // each weight byte is read once per launch) AND of the two activation rows (read by every CTA, so they stay in L2)
    // before it uses any of them - a launch of this kernel is one or two memory round trips long, and a load issued after
    // a wait would add its whole latency to that.  The activations by ordinary loads (see grid_dependency_wait).
    const uint4 z = make_uint4(0, 0, 0, 0);
    // whether this lane's 8 elements of step s lie inside K
    auto inside = [&](int s) { return !RAGGED || kbase + (size_t)s * 32 < (size_t)p.K; };
    uint4 wv[CH], wv2[SWIGLU ? CH : 1], al[CH], ah[CH];
    auto load_weights = [&](int s0) {
#pragma unroll
        for (int s = 0; s < CH; ++s)
            if (s0 + s < p.steps) {
                // 32 K positions = 64 B = 4 x 16 B per row and step
                wv[s] = inside(s0 + s) ? __ldcs(bw + (size_t)(s0 + s) * 4) : z;
                if (SWIGLU) wv2[s] = inside(s0 + s) ? __ldcs(bw2 + (size_t)(s0 + s) * 4) : z;
            }
    };
    // The warp's whole slice of the 8 weight rows is requested into L2 at once (a 128-byte line is two steps of a
    // row; the four lanes of a row name the same line and are merged): the batches below then find their weights
    // in L2 instead of each paying a round trip to HBM.  Under a programmatic dependent launch this happens while the
    // kernel before this one in the stream is still running - the weights do not depend on it, the activations do,
    // and nothing is READ before the wait (L2 is the point of coherence, so a line prefetched early cannot go stale).
    for (int s = 0; s < p.steps; s += 2) {
        if (!inside(s)) break;
        asm volatile("prefetch.global.L2 [%0];" ::"l"(bw + (size_t)s * 4));
        if (SWIGLU) asm volatile("prefetch.global.L2 [%0];" ::"l"(bw2 + (size_t)s * 4));
    }
    grid_dependency_wait();
    grid_launch_dependents();
    auto load_rows = [&](int s0, uint4 (&lo)[CH], uint4 (&hi)[CH]) {
#pragma unroll
        for (int s = 0; s < CH; ++s)
            if (s0 + s < p.steps) {
                lo[s] = lo_ok && inside(s0 + s) ? a_lo[(size_t)(s0 + s) * 4] : z;
                hi[s] = hi_ok && inside(s0 + s) ? a_hi[(size_t)(s0 + s) * 4] : z;
            }
    };
    auto multiply = [&](int s0, const uint4 (&lo)[CH], const uint4 (&hi)[CH]) {
#pragma unroll
        for (int s = 0; s < CH; ++s)
            if (s0 + s < p.steps) {
                // two k16 MMAs per step: the lane's first four K positions play (2j, 2j+1, 2j+8, 2j+9) of the first,
                // its last four of the second, in A and B alike
                mma_bf16_16816(acc, lo[s].x, hi[s].x, lo[s].y, hi[s].y, wv[s].x, wv[s].y);
                mma_bf16_16816(acc, lo[s].z, hi[s].z, lo[s].w, hi[s].w, wv[s].z, wv[s].w);
                if (SWIGLU) {
                    mma_bf16_16816(acc2, lo[s].x, hi[s].x, lo[s].y, hi[s].y, wv2[s].x, wv2[s].y);
                    mma_bf16_16816(acc2, lo[s].z, hi[s].z, lo[s].w, hi[s].w, wv2[s].z, wv2[s].w);
                }
            }
    };
    if (CH == 2 && !RAGGED && p.M > 4) {
        // short batches: the next batch's activations are requested ahead of this one's arithmetic, too (a LLaMA step of 16
        // sequences, 4 blocks, 300 us; without 314; a single row has little to wait for: a Soluzen step 254.5 us, with it 255.5)
        uint4 nl[CH], nh[CH];
        load_rows(0, al, ah);
        for (int s0 = 0; s0 < p.steps; s0 += 2 * CH) {
            load_weights(s0);
            load_rows(s0 + CH, nl, nh);
            multiply(s0, al, ah);
            load_weights(s0 + CH);
            load_rows(s0 + 2 * CH, al, ah);
            multiply(s0 + CH, nl, nh);
        }
    } else {
        for (int s0 = 0; s0 < p.steps; s0 += CH) {
            load_weights(s0);
            load_rows(s0, al, ah);
            multiply(s0, al, ah);
        }
    }
    // C fragment: acc[0], acc[1] = row g, columns 2j, 2j+1; acc[2], acc[3] = row g + 8
    s_part[warp][0][g][2 * j] = acc[0];
    s_part[warp][0][g][2 * j + 1] = acc[1];
    s_part[warp][0][g + 8][2 * j] = acc[2];
    s_part[warp][0][g + 8][2 * j + 1] = acc[3];
    if (SWIGLU) {
        s_part[warp][1][g][2 * j] = acc2[0];
        s_part[warp][1][g][2 * j + 1] = acc2[1];
        s_part[warp][1][g + 8][2 * j] = acc2[2];
        s_part[warp][1][g + 8][2 * j + 1] = acc2[3];
    }
    __syncthreads();
    if (threadIdx.x < 128) {
        const int row = threadIdx.x / 8, col = threadIdx.x % 8;
        float v = 0.f, u = 0.f;
        if (row < p.M) {
#pragma unroll
            for (int w = 0; w < SK_WARPS; ++w) {
                v += s_part[w][0][row][col];
                if (SWIGLU) u += s_part[w][1][row][col];
            }
            if (SWIGLU) v = activation_fast(p.act, v) * u;                // act(gate) * up
        }
        const int n = n0 + col;
        if (APPEND && n >= p.n_end[0]) {       // the same for the CTA's 8 columns: the ranges are multiples of 8
            skinny_append(p, row, n, v);
        } else if (row < p.M) {
            skinny_store<SWIGLU>(p, row, n, v);
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------
// The same for K a multiple of 256: CTAs that stay, two a multiprocessor, and take the groups of eight columns in turn.  A warp
// keeps its eighth of the activation rows in registers for all of them (the kernel above reads all rows again for every eight
// columns: with 16 rows that is as much as a weight) and has the next slice of its weight rows on the way into shared memory
// of its own while it multiplies one: 512 contiguous bytes of a row an instruction, where a fragment's own load is 64 bytes of
// eight rows each.  No warp waits for another but in the sum over warps, whose buffer alternates.
// What bounds it is HBM, after the few us until the first rows are there.  us with 1 / 16 rows, before and now, and what
// the weight takes at the copy bandwidth: 2048 -> 32000 26.0 / 33.9, 20.2 / 22.8 (20.1); 2048 -> 8512 9.6 / 11.6, 6.7 / 8.4
// (5.4); gated pair 2048 -> 5632 11.7 / 12.8, 9.0 / 10.0 (7.1); 2048 -> 2560 4.5 / 5.7, 3.5 / 5.0 (1.6).  Three slices of
// room instead of two: the same for the widest, 10 % slower for 2048 -> 4608; one CTA a multiprocessor with six: 12 - 40 %
// slower; slices asked for in L2 further ahead: 2 - 10 % slower.
// MULTI: K above 2048, in parts of which a warp holds one at a time, so that the rows are read again for every group, of which a CTA has
// few (2048 columns: one).
// ---------------------------------------------------------------------------------------------------------------
constexpr int WD_STAGES = 2, WD_STEPS = 8, WD_SLICE = 8 * WD_STEPS * 64;
constexpr int WD_SMEM = SK_WARPS * WD_STAGES * WD_SLICE, WD_CTAS = 2;

// HI: more than eight rows
template <bool GLU, bool HI, bool MULTI, bool APPEND>
__global__ void __launch_bounds__(SK_WARPS * 32, WD_CTAS)
gemm_wide_kernel(const SkinnyParams p) {
    constexpr int UNITS = GLU ? 2 : 1;                    // weights of a group: gate and up
    extern __shared__ __align__(128) uint8_t wd_smem[];
    __shared__ __align__(8) float s_part[2][UNITS][SK_WARPS][16][8];
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, g = lane / 4, j = lane % 4;
    const int groups = p.N / 8, mine = (groups - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
    const int parts = MULTI ? (p.steps + WD_STEPS - 1) / WD_STEPS : 1, n_slices = mine * parts * UNITS;
    const size_t kbase = (size_t)warp * p.steps * 32;
    auto steps_of = [&](int part) { return MULTI ? min(WD_STEPS, p.steps - part * WD_STEPS) : p.steps; };
    // Slices in the order group, part, weight: where slice u starts
    auto slice = [&](int u) {
        const int part = MULTI ? u / UNITS % parts : 0, i = u / UNITS / parts;
        const int n0 = ((int)blockIdx.x + i * (int)gridDim.x) * 8;
        return (GLU && u % 2 ? p.bt2 : p.bt) + (size_t)n0 * p.K + kbase + part * (WD_STEPS * 32);
    };
    const uint32_t ring = smem_u32(wd_smem) + warp * (WD_STAGES * WD_SLICE);
    // Row r's piece c lies at piece c ^ (4 for odd r): the eight lanes of a phase (two rows, four pieces) meet different banks
    auto fetch = [&](int u) {
        if (u < n_slices && lane < steps_of(MULTI ? u / UNITS % parts : 0) * 4) {
            const __nv_bfloat16* w = slice(u) + lane * 8;
            const uint32_t to = ring + u % WD_STAGES * WD_SLICE;
#pragma unroll
            for (int r = 0; r < 8; ++r) cp_async_16(to + r * 512 + ((lane ^ (r & 1) * 4) * 16), w + (size_t)r * p.K, 16);
        }
        cp_async_commit();
    };
    // The first slices are asked for in L2 beside the kernel ahead: the weights do not depend on it, and nothing is READ before the
    // wait.  A lane has a line of 64 elements of a row.
#pragma unroll
    for (int u = 0; u < WD_STAGES; ++u)
        if (u < n_slices && j * 64 < steps_of(MULTI ? u / UNITS % parts : 0) * 32) prefetch_l2(slice(u) + (size_t)g * p.K + j * 64);
    grid_dependency_wait();
    grid_launch_dependents();
#pragma unroll
    for (int u = 0; u < WD_STAGES - 1; ++u) fetch(u);
    const uint4 z = make_uint4(0, 0, 0, 0);
    const uint4* a_lo = reinterpret_cast<const uint4*>(p.a + (size_t)g * p.K + kbase) + j;
    const uint4* a_hi = reinterpret_cast<const uint4*>(p.a + (size_t)(g + 8) * p.K + kbase) + j;
    uint4 al[WD_STEPS], ah[HI ? WD_STEPS : 1];
    ah[0] = z;
    auto load_rows = [&](int part) {
        const int n = steps_of(part);
#pragma unroll
        for (int s = 0; s < WD_STEPS; ++s) {
            al[s] = s < n && g < p.M ? a_lo[(part * WD_STEPS + s) * 4] : z;
            if (HI) ah[HI ? s : 0] = s < n && g + 8 < p.M ? a_hi[(part * WD_STEPS + s) * 4] : z;
        }
    };
    load_rows(0);
    for (int i = 0, u = 0; i < mine; ++i) {
        const int buf = i & 1;
        float acc[UNITS][2][4];                           // two chains of MMAs each
#pragma unroll
        for (int k = 0; k < UNITS; ++k)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[k][0][c] = acc[k][1][c] = 0.f;
        for (int part = 0; part < parts; ++part) {
            const int n = steps_of(part);
#pragma unroll
            for (int k = 0; k < UNITS; ++k, ++u) {
                fetch(u + WD_STAGES - 1);
                cp_async_wait<WD_STAGES - 1>();
                __syncwarp();
                const uint8_t* at = wd_smem + warp * (WD_STAGES * WD_SLICE) + u % WD_STAGES * WD_SLICE + g * 512;
#pragma unroll
                for (int s = 0; s < WD_STEPS; ++s)
                    if (s < n) {
                        const uint4 w = *reinterpret_cast<const uint4*>(at + ((s * 4 + j) ^ (g & 1) * 4) * 16);
                        mma_bf16_16816(acc[k][0], al[s].x, ah[HI ? s : 0].x, al[s].y, ah[HI ? s : 0].y, w.x, w.y);
                        mma_bf16_16816(acc[k][1], al[s].z, ah[HI ? s : 0].z, al[s].w, ah[HI ? s : 0].w, w.z, w.w);
                    }
                __syncwarp();                             // the slice is read before the next fetch overwrites it
            }
            if (MULTI && (part + 1 < parts || i + 1 < mine)) load_rows(part + 1 < parts ? part + 1 : 0);
        }
#pragma unroll
        for (int k = 0; k < UNITS; ++k) {
            float (*sums)[8] = s_part[buf][k][warp];
            *reinterpret_cast<float2*>(&sums[g][2 * j]) = make_float2(acc[k][0][0] + acc[k][1][0], acc[k][0][1] + acc[k][1][1]);
            if (HI) *reinterpret_cast<float2*>(&sums[g + 8][2 * j]) = make_float2(acc[k][0][2] + acc[k][1][2], acc[k][0][3] + acc[k][1][3]);
        }
        __syncthreads();
        // four of the warps, in turn; the others go on, as far as the next sum
        const int t = (int)threadIdx.x - buf * 128;
        if (t >= 0 && t < 128) {
            const int row = t / 8, n = ((int)blockIdx.x + i * (int)gridDim.x) * 8 + t % 8;
            float v = 0.f, up = 0.f;
            if (row < p.M) {
#pragma unroll
                for (int w = 0; w < SK_WARPS; ++w) {
                    v += s_part[buf][0][w][row][t % 8];
                    if (GLU) up += s_part[buf][UNITS - 1][w][row][t % 8];
                }
                if (GLU) v = activation_fast(p.act, v) * up;
            }
            if (APPEND && n >= p.n_end[0]) skinny_append(p, row, n, v);
            else if (row < p.M) skinny_store<GLU>(p, row, n, v);
        }
    }
    cp_async_wait<0>();
}

static int skinny_check(const char* what, const void* a, const void* bt, int M, int N, int K) {
    if (!a || !bt) return fail(BN_ERR_INVALID_ARG, "%s: null pointer", what);
    if (M <= 0 || M > 16) return fail(BN_ERR_UNSUPPORTED, "%s: M=%d (1..16 rows)", what, M);
    if (N <= 0 || N % 8) return fail(BN_ERR_UNSUPPORTED, "%s: N=%d must be a positive multiple of 8", what, N);
    if (K <= 0 || K % 8 || K > SK_WARPS * 32 * SK_MAX_STEPS)
        return fail(BN_ERR_UNSUPPORTED, "%s: K=%d must be a multiple of 8, at most %d", what, K, SK_WARPS * 32 * SK_MAX_STEPS);
    if ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(bt)) & 15)
        return fail(BN_ERR_INVALID_ARG, "%s: a/bt must be 16-byte aligned", what);
    return require_sm100();
}

// Which kernel.  Of the first: up to two CTAs per SM run fastest with 8 steps in flight, more with four per SM and 2; the gated pair
// holds two weights and runs with 2.
template <bool GLU, bool APPEND>
static int skinny_launch(const SkinnyParams& p, cudaStream_t st, const char* what) {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // us before and now, the kernel that stays second.  Gated pairs: 2048 -> 2048 5.4, 4.1, -> 3072 6.0, 6.4 (three CTAs a multiprocessor
    // hold all groups at once), -> 5632 11.7, 9.0.  Others with 8 rows: 2048 -> 256 2.2, 2.1, -> 4608 5.4, 4.9, 4096 -> 2048 5.4, 4.6,
    // 7424 -> 2048 8.6, 7.3, but 1024 -> 4608 3.3, 3.5 (1024 -> 6144, in two waves, 5.0, 4.1); with 16 rows the groups have
    // to share CTAs before the rows kept pay: 2048 -> 512 2.6, 3.0, -> 2048 4.0, 4.1, -> 2560 5.7, 5.0
    const int groups = p.N / 8;
    const bool wide = GLU ? groups <= 2 * sms || groups > 3 * sms
                          : groups > 4 * sms || (p.K >= 1280 && (p.M <= 8 || p.K > 2048 || groups > 2 * sms));
    if (wide && p.K % (SK_WARPS * 32) == 0) {
        auto run = [&](auto kernel) {
            if (int rc = allow_smem(kernel, WD_SMEM, what)) return rc;
            launch_dependent(kernel, (unsigned)(groups < WD_CTAS * sms ? groups : WD_CTAS * sms), SK_WARPS * 32, WD_SMEM, st, p);
            return launch_status(what);
        };
        if (p.steps > WD_STEPS) return p.M > 8 ? run(gemm_wide_kernel<GLU, true, true, APPEND>) : run(gemm_wide_kernel<GLU, false, true, APPEND>);
        return p.M > 8 ? run(gemm_wide_kernel<GLU, true, false, APPEND>) : run(gemm_wide_kernel<GLU, false, false, APPEND>);
    }
    const bool deep = !GLU && p.N / 8 <= 2 * sms;
    if (p.K % (SK_WARPS * 32)) launch_dependent(gemm_skinny_kernel<GLU, 2, APPEND, true>, p.N / 8, SK_WARPS * 32, 0, st, p);
    else if (deep) launch_dependent(gemm_skinny_kernel<GLU, GLU ? 2 : 8, APPEND>, p.N / 8, SK_WARPS * 32, 0, st, p);
    else launch_dependent(gemm_skinny_kernel<GLU, 2, APPEND>, p.N / 8, SK_WARPS * 32, 0, st, p);
    return launch_status(what);
}

}  // namespace bn

using namespace bn;

extern "C" int bn_gemm_bf16_nt_skinny(const void* a, const void* bt, int M, int N, int K, void* out0, int n0, void* out1,
                                      int n1, void* out2, bn_stream_t stream) {
    const char* what = "bn_gemm_bf16_nt_skinny";
    if (int rc = skinny_check(what, a, bt, M, N, K)) return rc;
    if (!out0 || n0 <= 0 || n0 > N || n0 % 8 || n1 < 0 || n1 % 8 || n0 + n1 > N || (n1 > 0 && !out1) ||
        (n0 + n1 < N && !out2))
        return fail(BN_ERR_INVALID_ARG, "%s: column ranges %d + %d of %d need their outputs (multiples of 8)", what, n0, n1, N);
    SkinnyParams p{};
    p.a = static_cast<const __nv_bfloat16*>(a);
    p.bt = static_cast<const __nv_bfloat16*>(bt);
    p.bt2 = nullptr;
    p.out[0] = static_cast<__nv_bfloat16*>(out0);
    p.out[1] = static_cast<__nv_bfloat16*>(out1);
    p.out[2] = static_cast<__nv_bfloat16*>(out2);
    p.n_end[0] = n0; p.n_end[1] = n0 + n1; p.n_end[2] = N;
    p.ld[0] = n0; p.ld[1] = n1; p.ld[2] = N - n0 - n1;
    p.M = M; p.N = N; p.K = K; p.steps = (K + SK_WARPS * 32 - 1) / (SK_WARPS * 32);
    return skinny_launch<false, false>(p, as_stream(stream), what);
}

static int skinny_f32(const char* what, const void* a, const void* bt, int M, int N, int K, float* out, bool rounded, bn_stream_t stream) {
    if (int rc = skinny_check(what, a, bt, M, N, K)) return rc;
    if (!out) return fail(BN_ERR_INVALID_ARG, "%s: null pointer", what);
    SkinnyParams p{};
    p.a = static_cast<const __nv_bfloat16*>(a);
    p.bt = static_cast<const __nv_bfloat16*>(bt);
    p.out32 = out; p.rounded = rounded;
    p.n_end[0] = p.n_end[1] = p.n_end[2] = N;
    p.M = M; p.N = N; p.K = K; p.steps = (K + SK_WARPS * 32 - 1) / (SK_WARPS * 32);
    return skinny_launch<false, false>(p, as_stream(stream), what);
}

extern "C" int bn_gemm_bf16_nt_skinny_f32(const void* a, const void* bt, int M, int N, int K, float* out, bn_stream_t stream) {
    return skinny_f32("bn_gemm_bf16_nt_skinny_f32", a, bt, M, N, K, out, false, stream);
}

extern "C" int bn_gemm_bf16_nt_skinny_widened(const void* a, const void* bt, int M, int N, int K, float* out, bn_stream_t stream) {
    return skinny_f32("bn_gemm_bf16_nt_skinny_widened", a, bt, M, N, K, out, true, stream);
}

extern "C" int bn_gemm_bias_act_bf16_nt_skinny(const void* a, const void* bt, const float* bias, void* out, int M, int N, int K,
                                               int act, bn_stream_t stream) {
    const char* what = "bn_gemm_bias_act_bf16_nt_skinny";
    if (int rc = skinny_check(what, a, bt, M, N, K)) return rc;
    if (!out || act < 0 || act > BN_ACT_LAST) return fail(BN_ERR_INVALID_ARG, "%s: bad argument", what);
    SkinnyParams p{};
    p.a = static_cast<const __nv_bfloat16*>(a);
    p.bt = static_cast<const __nv_bfloat16*>(bt);
    p.out[0] = static_cast<__nv_bfloat16*>(out);
    p.n_end[0] = p.n_end[1] = p.n_end[2] = N;
    p.ld[0] = N;
    p.bias = bias; p.act = act;
    p.M = M; p.N = N; p.K = K; p.steps = (K + SK_WARPS * 32 - 1) / (SK_WARPS * 32);
    return skinny_launch<false, false>(p, as_stream(stream), what);
}

extern "C" int bn_gemm_act_mul_bf16_nt_skinny(const void* a, const void* bt, const void* mul, int64_t mul_ld, void* out, int M,
                                              int N, int K, int act, bn_stream_t stream) {
    const char* what = "bn_gemm_act_mul_bf16_nt_skinny";
    if (int rc = skinny_check(what, a, bt, M, N, K)) return rc;
    if (!mul || !out || mul_ld < N || act < 0 || act > BN_ACT_LAST) return fail(BN_ERR_INVALID_ARG, "%s: bad argument", what);
    SkinnyParams p{};
    p.a = static_cast<const __nv_bfloat16*>(a);
    p.bt = static_cast<const __nv_bfloat16*>(bt);
    p.out[0] = static_cast<__nv_bfloat16*>(out);
    p.n_end[0] = p.n_end[1] = p.n_end[2] = N;
    p.ld[0] = N;
    p.mul = static_cast<const __nv_bfloat16*>(mul); p.mul_ld = mul_ld; p.act = act;
    p.M = M; p.N = N; p.K = K; p.steps = (K + SK_WARPS * 32 - 1) / (SK_WARPS * 32);
    return skinny_launch<false, false>(p, as_stream(stream), what);
}

extern "C" int bn_gemm_glu_bf16_nt_skinny(const void* x, const void* gate_t, const void* up_t, void* h, int M, int inter,
                                          int K, int act, bn_stream_t stream) {
    const char* what = "bn_gemm_glu_bf16_nt_skinny";
    if (int rc = skinny_check(what, x, gate_t, M, inter, K)) return rc;
    if (!up_t || !h || (reinterpret_cast<uintptr_t>(up_t) & 15)) return fail(BN_ERR_INVALID_ARG, "%s: null or misaligned pointer", what);
    if (act < 0 || act > BN_ACT_LAST) return fail(BN_ERR_INVALID_ARG, "%s: activation %d", what, act);
    SkinnyParams p{};
    p.a = static_cast<const __nv_bfloat16*>(x);
    p.bt = static_cast<const __nv_bfloat16*>(gate_t);
    p.bt2 = static_cast<const __nv_bfloat16*>(up_t);
    p.out[0] = static_cast<__nv_bfloat16*>(h);
    p.n_end[0] = p.n_end[1] = p.n_end[2] = inter;
    p.ld[0] = inter;
    p.act = act;
    p.M = M; p.N = inter; p.K = K; p.steps = (K + SK_WARPS * 32 - 1) / (SK_WARPS * 32);
    return skinny_launch<true, false>(p, as_stream(stream), what);
}

extern "C" int bn_gemm_swiglu_bf16_nt_skinny(const void* x, const void* gate_t, const void* up_t, void* h, int M, int inter,
                                             int K, bn_stream_t stream) {
    return bn_gemm_glu_bf16_nt_skinny(x, gate_t, up_t, h, M, inter, K, BN_ACT_SILU, stream);
}

extern "C" int bn_gemm_qkv_append_bf16_skinny(const void* x, const void* wqkv_t, int M, int hidden, int Hq, int Hkv, int D,
                                              void* q_out, void* pool, int64_t pool_pages, const int32_t* page_table,
                                              int max_pages, const int32_t* seq_ids, const int32_t* positions, float theta,
                                              bn_stream_t stream) {
    const char* what = "bn_gemm_qkv_append_bf16_skinny";
    if (Hq <= 0 || Hkv <= 0 || D <= 0 || D % 8)
        return fail(BN_ERR_INVALID_ARG, "%s: bad head shape Hq=%d Hkv=%d D=%d (D a multiple of 8)", what, Hq, Hkv, D);
    const int N = (Hq + 2 * Hkv) * D;
    if (int rc = skinny_check(what, x, wqkv_t, M, N, hidden)) return rc;
    if (!q_out || !pool || !page_table || !seq_ids || !positions || max_pages <= 0 || pool_pages <= 0)
        return fail(BN_ERR_INVALID_ARG, "%s: null pointer or empty cache", what);
    SkinnyParams p{};
    p.a = static_cast<const __nv_bfloat16*>(x);
    p.bt = static_cast<const __nv_bfloat16*>(wqkv_t);
    p.out[0] = static_cast<__nv_bfloat16*>(q_out);
    p.n_end[0] = Hq * D; p.n_end[1] = (Hq + Hkv) * D; p.n_end[2] = N;
    p.ld[0] = Hq * D;
    p.M = M; p.N = N; p.K = hidden; p.steps = (hidden + SK_WARPS * 32 - 1) / (SK_WARPS * 32);
    p.pool = static_cast<__nv_bfloat16*>(pool);
    p.page_table = page_table; p.seq_ids = seq_ids; p.positions = positions;
    p.pool_pages = pool_pages; p.max_pages = max_pages; p.Hkv = Hkv; p.D = D; p.theta = theta;
    return skinny_launch<false, true>(p, as_stream(stream), what);
}
