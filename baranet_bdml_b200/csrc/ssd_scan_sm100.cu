// The selective state-space recurrence of a prompt portion in chunks of 128 tokens on tcgen05, for 64 values a head and a state of
// 128 (bf16 inputs): what ssd_scan_kernel computes with warp-level MMAs, whose issue slots bound it (2830 instructions a warp and 64
// tokens, of which 456 were MMAs and the loads of their operands).
//
// A CTA has a head of a sequence and walks its chunks.  With c_i the running sum of the chunk's log decays and S (128 x 64, state x
// value) the state before the chunk, five products a chunk, fp32 sums in tensor memory:
//   G  = C B^T                            128 x 128, K = 128
//   Y2 = C S                              128 x 64      y_i = Y1_i + e^{c_i} Y2_i + D x_i
//   U  = B^T (w x)                        128 x 64      S' = e^{c_last} S + U,  w_j = e^{c_last - c_j} dt_j
//   Y1 = M x,  M_ij = G_ij e^{c_i - c_j} dt_j  (j <= i)
// S, w x and M are fp32 quantities: each goes in as TWO bf16 numbers, its rounding and the remainder (16 bits), so three of the
// products run twice; x, B and C are bf16 as they come.  M goes from tensor memory to tensor memory through the registers of the
// thread that has its row; S' lives in registers (a thread: one of the 128 states, 32 of the values), its two parts in shared memory.
//
// Exponents are sums over tokens from i back to j.  They are taken inside blocks of 32 tokens: c is summed within a block, so that the
// difference of two of them is exact to the block's own size, and outside the diagonal blocks e^{c_i - c_j} is a factor of the row,
// e^{from the end of j's block to i}, times one of the column, e^{from j to the end of its block} dt_j, both at most 1: no exponential
// per element there.
//
// Warps 0-7: the rest of the arithmetic (thread = token row or state row, half of the columns); warp 8: TMA of tiles and outputs; warp 9:
// MMAs; warp 10: decays.  G, Y2 and U of the next chunk run while this one's outputs are finished and its own M is worked out.  160 KB of
// tiles, one CTA a multiprocessor.  A chunk takes about 4200 cycles, of which 3750 are shared memory's at 128 bytes a cycle (480 KB:
// tiles in 80, the five products' operands 288, parts, x and outputs through the threads 112), MMAs 2050.
// 8 x 2048 tokens, 64 heads: 187 us (ssd_scan_kernel 442); 1 x 2048 43 (285); 3 x 333 23 (65); 1 x 128 6.5 (22).
// On the way: a and dt loaded and summed by the TMA warp behind its waits 206 us; sixteen warps with a quarter of the columns each 242.
//
// A token with an x that is not finite reaches the tokens before it in its 16 at most, as in the warp-level form: the MMAs of 16 columns
// of M leave the rows before them alone (disabled output lanes).
#include "common.cuh"
#include "hybrid.cuh"
#include "mamba2.cuh"
#include "ptx.cuh"
#include "tcgen05.cuh"
#include "tma.cuh"

namespace bn {

using namespace ptx;

constexpr int ST_Q = 128, ST_N = 128, ST_P = 64, ST_WORK = 256, ST_THREADS = ST_WORK + 96;
constexpr int ST_HALF = ST_Q * 128;                                   // 128 rows of 128 bytes
constexpr int ST_TILES = 5 * ST_HALF;                                 // C (two halves of 64 columns), B (two), x
constexpr int ST_S = 2 * ST_TILES, ST_WX = ST_S + 2 * ST_HALF, ST_ARRAYS = ST_WX + 2 * ST_HALF;
// of a chunk: loc_i (running sum within the block, log2), dt_j, the column's factor, the blocks' sums.  dt_j stays a factor: in the
// exponent it would be rounded to the spacing of a sum of 32 decays, and could not be negative.
struct StArrays { float loc[ST_Q], dt[ST_Q], col[ST_Q - 32], total[4]; };
struct StTail {
    StArrays arrays[2];
    uint64_t full[2], empty[2], g, ops, u, m, y, out;
    uint32_t tmem;
    int abort;
};
constexpr int ST_SMEM = ST_ARRAYS + (int)sizeof(StTail);              // all there is, less 144 bytes: no slack for an alignment
static_assert(ST_SMEM <= 227 * 1024, "shared memory");
constexpr uint32_t ST_G = 0, ST_MH = 128, ST_ML = 192, ST_Y1 = 256, ST_U = 320, ST_Y2 = 384;   // columns of tensor memory (two of Y2)

struct StParams {
    SsmScanParams s;
    int* error_word;
};

// D[tmem] (+)= A[tmem] B, of the rows from 16 r on only
__device__ __forceinline__ void mma_ts_rows(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate, int r) {
    const int lanes = r * 16;                                         // lanes 0 .. lanes - 1 stay as they are
    uint32_t off[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) off[i] = lanes >= 32 * (i + 1) ? 0xffffffffu : lanes > 32 * i ? 0xffffu : 0u;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %6, %7, %8}, p;\n\t}"
        ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(off[0]), "r"(off[1]), "r"(off[2]), "r"(off[3])
        : "memory");
}

__device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& lo) {
    hi = pack_bf16(a, b);
    lo = pack_bf16(a - bf16_lo(hi), b - bf16_hi(hi));
}

__global__ void __launch_bounds__(ST_THREADS, 1) ssd_scan_tc_kernel(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ CUtensorMap tmap_y,
                                                                     const __grid_constant__ StParams q) {
    extern __shared__ __align__(1024) uint8_t base[];
    StTail& tail = *reinterpret_cast<StTail*>(base + ST_ARRAYS);
    uint64_t (&bar_full)[2] = tail.full, (&bar_empty)[2] = tail.empty;
    uint64_t &bar_g = tail.g, &bar_ops = tail.ops, &bar_u = tail.u, &bar_m = tail.m, &bar_y = tail.y, &bar_out = tail.out;
    int& s_abort = tail.abort;
    StArrays* arrays = tail.arrays;
    const SsmScanParams& p = q.s;
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    const uint32_t smem0 = smem_u32(base);
    if (smem0 & 1023) {                                               // (the tiles' swizzle needs it; uniform, and not seen)
        grid_dependency_wait();
        if (tid == 0) atomicExch(q.error_word, BN_ERR_TIMEOUT);
        return;
    }
    const int h = blockIdx.x % p.H, b = blockIdx.x / p.H, grp = h / (p.H / p.G), chunks = (p.S + ST_Q - 1) / ST_Q;
    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(smem_u32(&bar_full[i]), 2);                     // the tiles, and the arrays
            mbar_init(smem_u32(&bar_empty[i]), 1);
        }
        mbar_init(smem_u32(&bar_g), 1);
        mbar_init(smem_u32(&bar_ops), ST_WORK / 32);           // a warp arrives once: an arrival a thread is a queue at one address
        mbar_init(smem_u32(&bar_u), 1);
        mbar_init(smem_u32(&bar_m), ST_WORK / 32);
        mbar_init(smem_u32(&bar_y), 1);
        mbar_init(smem_u32(&bar_out), ST_WORK / 32);
        s_abort = 0;
        fence_mbar_init();
    }
    if (warp == 9) {
        tc::tmem_alloc(smem_u32(&tail.tmem), 512);
        tc::tmem_relinquish();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tail.tmem;
    grid_dependency_wait();
    grid_launch_dependents();

    if (warp == 8) {
        // ------------------------------------------------ the next chunk's tiles, outputs on their way
        if (lane == 0) {
            prefetch_tensormap(&tmap);
            prefetch_tensormap(&tmap_y);
            const int inner = p.H * p.P, cx = h * p.P, cb = inner + grp * p.N, cc = cb + p.G * p.N;
            for (int k = 0; k < chunks + 2; ++k) {
                const int buf = k & 1, t0 = k * ST_Q;
                if (!mbar_wait(smem_u32(&bar_empty[buf]), ((k >> 1) & 1u) ^ 1u, &s_abort)) break;
                const uint32_t full = smem_u32(&bar_full[buf]), tiles = smem0 + buf * ST_TILES;
                if (k < chunks) {
                    mbar_arrive_expect_tx(full, ST_TILES);
                    tma_load_3d(tiles, &tmap, cc, t0, b, full);
                    tma_load_3d(tiles + ST_HALF, &tmap, cc + 64, t0, b, full);
                    tma_load_3d(tiles + 2 * ST_HALF, &tmap, cb, t0, b, full);
                    tma_load_3d(tiles + 3 * ST_HALF, &tmap, cb + 64, t0, b, full);
                }
                if (k >= 2) {                                         // the outputs of two chunks ago lie where their x did
                    if (!mbar_wait(smem_u32(&bar_out), k & 1u, &s_abort)) break;
                    tma_store_3d(&tmap_y, tiles + 4 * ST_HALF, cx, t0 - 2 * ST_Q, b);
                    bulk_commit_group();
                    bulk_wait_group_read0();
                }
                if (k < chunks) tma_load_3d(tiles + 4 * ST_HALF, &tmap, cx, t0, b, full);
            }
        }
        __syncwarp();
    } else if (warp == 10) {
        // ------------------------------------------------ the next chunk's decays and step sizes
        for (int k = 0; k < chunks; ++k) {
            float a[4], d[4], loc[4], s = 0.f;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int t = k * ST_Q + lane * 4 + e;
                const int64_t at = ((int64_t)b * p.S + t) * p.H + h;
                a[e] = t < p.S ? p.a[at] : 0.f;                       // beyond the sequence: no decay, steps of 0
                d[e] = t < p.S ? p.dt[at] : 0.f;
            }
            // running sums within blocks of 32 tokens = 8 lanes, in log2
#pragma unroll
            for (int e = 0; e < 4; ++e) { s += a[e] * 1.44269504088896f; loc[e] = s; }
            float before = s;
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) {
                const float u = __shfl_up_sync(0xffffffffu, before, o);
                if (lane % 8 >= o) before += u;
            }
            const float total = __shfl_sync(0xffffffffu, before, lane / 8 * 8 + 7);
            before -= s;
            float own[4], col[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                own[e] = before + loc[e];
                col[e] = exp2f(total - own[e]) * d[e];
            }
            if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_empty[k & 1]), ((k >> 1) & 1u) ^ 1u, &s_abort))) break;
            StArrays& w = arrays[k & 1];
            store4(w.loc + lane * 4, own);
            store4(w.dt + lane * 4, d);
            if (lane < 24) store4(w.col + lane * 4, col);
            if (lane % 8 == 7) w.total[lane / 8] = total;
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bar_full[k & 1]));
        }
    } else if (warp == 9) {
        // ------------------------------------------------ MMAs
        // MN-major operands: rows are k.  x, S and w x have 64 columns (values), B^T 128 (states): the second 64 lie ST_HALF further on
        constexpr uint32_t I_G = tc::idesc_bf16(128, 128, 0), I_N = tc::idesc_bf16(128, 64, 1), I_U = I_N | 1u << 15;
        const uint64_t d0 = tc::smem_desc_sw128(0), dT = (d0 & ~((uint64_t)0x3fff << 16)) | (uint64_t)(ST_HALF >> 4) << 16;
        auto at = [](uint64_t d, uint32_t addr) { return d + (uint64_t)(addr >> 4); };
        const uint32_t uS = smem0 + ST_S, uW = smem0 + ST_WX;
        auto issue_g = [&](int k) {
            const uint32_t uC = smem0 + (k & 1) * ST_TILES, uB = uC + 2 * ST_HALF;
            if (!mbar_wait(smem_u32(&bar_full[k & 1]), (k >> 1) & 1u, &s_abort)) return false;
            if (elect_one()) {
                tc::fence_after_sync();
#pragma unroll
                for (int kk = 0; kk < 8; ++kk)
                    tc::mma_ss(tmem + ST_G, at(d0, uC + kk / 4 * ST_HALF + kk % 4 * 32), at(d0, uB + kk / 4 * ST_HALF + kk % 4 * 32), I_G, kk > 0);
                tc::commit(smem_u32(&bar_g));
            }
            __syncwarp();
            return true;
        };
        bool ok = issue_g(0);
        for (int k = 0; ok && k < chunks; ++k) {
            const uint32_t uC = smem0 + (k & 1) * ST_TILES, uB = uC + 2 * ST_HALF, uX = uC + 4 * ST_HALF;
            ok = mbar_wait(smem_u32(&bar_ops), k & 1u, &s_abort);     // S and w x are there, Y2 of two chunks ago has been read
            if (!ok) break;
            if (elect_one()) {
                tc::fence_after_sync();
#pragma unroll
                for (int part = 1; part >= 0; --part)
#pragma unroll
                    for (int kk = 0; kk < 8; ++kk)
                        tc::mma_ss(tmem + ST_Y2 + (k & 1) * 64, at(d0, uC + kk / 4 * ST_HALF + kk % 4 * 32), at(d0, uS + part * ST_HALF + kk * 2048), I_N, part == 0 || kk > 0);
#pragma unroll
                for (int part = 1; part >= 0; --part)
#pragma unroll
                    for (int kk = 0; kk < 8; ++kk)
                        tc::mma_ss(tmem + ST_U, at(dT, uB + kk * 2048), at(d0, uW + part * ST_HALF + kk * 2048), I_U, part == 0 || kk > 0);
                tc::commit(smem_u32(&bar_u));
            }
            __syncwarp();
            ok = mbar_wait(smem_u32(&bar_m), k & 1u, &s_abort);       // M is there, and G has been read
            if (!ok) break;
            if (elect_one()) {
                tc::fence_after_sync();
#pragma unroll
                for (int part = 1; part >= 0; --part)
#pragma unroll
                    for (int kk = 0; kk < 8; ++kk)
                        mma_ts_rows(tmem + ST_Y1, tmem + (part ? ST_ML : ST_MH) + kk * 8, at(d0, uX + kk * 2048), I_N, part == 0 || kk > 0, kk);
                tc::commit(smem_u32(&bar_y));
                tc::commit(smem_u32(&bar_empty[k & 1]));
            }
            __syncwarp();
            if (k + 1 < chunks) ok = issue_g(k + 1);
        }
    } else {
        // ------------------------------------------------ a row of tokens (or of the state) each, half of the columns
        const int rb = warp % 4, row = rb * 32 + lane, hf = warp / 4, slot = p.seq_ids ? p.seq_ids[b] : b;
        const uint32_t lanes = (uint32_t)(rb * 32) << 16;
        const float D = p.D[h];
        float* state = p.state + (((int64_t)slot * p.H + h) * ST_P + hf * 32) * ST_N + row;
        float st[32];
#pragma unroll
        for (int e = 0; e < 32; ++e) st[e] = state[(int64_t)e * ST_N];
        auto chunk_of = [&](int c) { return row * 128 + (((hf * 4 + c) ^ (row & 7)) << 4); };      // 8 values of a row of a tile
        auto put_state = [&]() {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                uint32_t hi[4], lo[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) split2(st[c * 8 + 2 * e], st[c * 8 + 2 * e + 1], hi[e], lo[e]);
                *reinterpret_cast<uint4*>(base + ST_S + chunk_of(c)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                *reinterpret_cast<uint4*>(base + ST_S + ST_HALF + chunk_of(c)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            }
        };
        put_state();
        // w x of a chunk in two parts; what its outputs need later stays with the thread
        struct Tokens { uint4 x[4]; float from_start, decay; } now, next;
        auto put_tokens = [&](Tokens& tk, int k) {
            const StArrays& w = arrays[k & 1];
            if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_full[k & 1]), (k >> 1) & 1u, &s_abort))) return false;
            float before = 0.f, after = 0.f, sum = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float t = w.total[i];
                before += i < rb ? t : 0.f;
                after += i > rb ? t : 0.f;
                sum += t;
            }
            const float weight = exp2f(w.total[rb] - w.loc[row] + after) * w.dt[row];
            tk.from_start = exp2f(w.loc[row] + before);
            tk.decay = exp2f(sum);
            const uint8_t* xt = base + (k & 1) * ST_TILES + 4 * ST_HALF;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                tk.x[c] = *reinterpret_cast<const uint4*>(xt + chunk_of(c));
                const uint32_t v[4] = {tk.x[c].x, tk.x[c].y, tk.x[c].z, tk.x[c].w};
                uint32_t hi[4], lo[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) split2(bf16_lo(v[e]) * weight, bf16_hi(v[e]) * weight, hi[e], lo[e]);
                *reinterpret_cast<uint4*>(base + ST_WX + chunk_of(c)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                *reinterpret_cast<uint4*>(base + ST_WX + ST_HALF + chunk_of(c)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            }
            return true;
        };
        auto hand_over = [&]() {                                       // w x and the state's parts, to the MMAs
            fence_proxy_async_smem();
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bar_ops));
        };
        bool ok = put_tokens(now, 0);
        if (ok) hand_over();
        for (int k = 0; ok && k < chunks; ++k) {
            const StArrays& w = arrays[k & 1];
            const float loc = w.loc[row];
            // M: blocks of 32 columns, up to the diagonal
            ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_g), k & 1u, &s_abort));
            if (!ok) break;
            tc::fence_after_sync();
#pragma unroll 1
            for (int i = 0; i < 2; ++i) {
                const int cb = hf + i * 2;
                uint32_t hi[16], lo[16];
                if (cb > rb) break;                                    // those MMAs leave these rows alone
                uint32_t g[32];
                tc::ld32(tmem + lanes + ST_G + cb * 32, g);
                tc::wait_ld(g);
                if (cb < rb) {
                    const float4* factors = reinterpret_cast<const float4*>(w.col) + cb * 8;
                    float between = 0.f;
#pragma unroll
                    for (int c = 1; c < 3; ++c) between += c > cb && c < rb ? w.total[c] : 0.f;
                    const float r = exp2f(loc + between);
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const float4 f = factors[e];
                        split2(__uint_as_float(g[4 * e]) * (r * f.x), __uint_as_float(g[4 * e + 1]) * (r * f.y), hi[2 * e], lo[2 * e]);
                        split2(__uint_as_float(g[4 * e + 2]) * (r * f.z), __uint_as_float(g[4 * e + 3]) * (r * f.w), hi[2 * e + 1], lo[2 * e + 1]);
                    }
                } else {
                    const float4 *locs = reinterpret_cast<const float4*>(w.loc) + cb * 8, *steps = reinterpret_cast<const float4*>(w.dt) + cb * 8;
                    auto element = [&](int j, float l, float d) { return j <= lane ? __uint_as_float(g[j]) * (ex2(loc - l) * d) : 0.f; };
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const float4 l = locs[e], d = steps[e];
                        split2(element(4 * e, l.x, d.x), element(4 * e + 1, l.y, d.y), hi[2 * e], lo[2 * e]);
                        split2(element(4 * e + 2, l.z, d.z), element(4 * e + 3, l.w, d.w), hi[2 * e + 1], lo[2 * e + 1]);
                    }
                }
                tc::st16(tmem + lanes + ST_MH + cb * 16, hi);
                tc::st16(tmem + lanes + ST_ML + cb * 16, lo);
            }
            tc::wait_st();
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bar_m));
            // the state behind the chunk
            ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_u), k & 1u, &s_abort));
            if (!ok) break;
            tc::fence_after_sync();
            {
                uint32_t u[32];
                tc::ld32(tmem + lanes + ST_U + hf * 32, u);
                tc::wait_ld(u);
#pragma unroll
                for (int e = 0; e < 32; ++e) st[e] = fmaf(now.decay, st[e], __uint_as_float(u[e]));
            }
            // the next chunk's operands ahead of this one's outputs, so that the MMAs go on (Y2 has read the state's parts before)
            if (k + 1 < chunks) {
                put_state();
                if (!(ok = put_tokens(next, k + 1))) break;
                hand_over();
            }
            // outputs
            ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_y), k & 1u, &s_abort));
            if (!ok) break;
            tc::fence_after_sync();
            uint8_t* out = base + (k & 1) * ST_TILES + 4 * ST_HALF;     // in place of x, from where the copies leave
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                uint32_t y1[16], y2[16], o[8];
                tc::ld16(tmem + lanes + ST_Y1 + hf * 32 + i * 16, y1);
                tc::ld16(tmem + lanes + ST_Y2 + (k & 1) * 64 + hf * 32 + i * 16, y2);
                tc::wait_ld(y1);
                tc::wait_ld(y2);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const uint4& xc = now.x[i * 2 + e / 4];
                    const uint32_t v = e % 4 == 0 ? xc.x : e % 4 == 1 ? xc.y : e % 4 == 2 ? xc.z : xc.w;
                    o[e] = pack_bf16(fmaf(D, bf16_lo(v), fmaf(now.from_start, __uint_as_float(y2[2 * e]), __uint_as_float(y1[2 * e]))),
                                     fmaf(D, bf16_hi(v), fmaf(now.from_start, __uint_as_float(y2[2 * e + 1]), __uint_as_float(y1[2 * e + 1]))));
                }
                *reinterpret_cast<uint4*>(out + chunk_of(i * 2)) = make_uint4(o[0], o[1], o[2], o[3]);
                *reinterpret_cast<uint4*>(out + chunk_of(i * 2 + 1)) = make_uint4(o[4], o[5], o[6], o[7]);
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bar_out));
            tc::fence_before_sync();
            now = next;
        }
        if (ok)
#pragma unroll
            for (int e = 0; e < 32; ++e) state[(int64_t)e * ST_N] = st[e];
    }
    // common exit: everybody arrives here (all waits are bounded), then TMEM is freed
    tc::fence_before_sync();
    __syncthreads();
    if (tid == 0 && s_abort) atomicExch(q.error_word, BN_ERR_TIMEOUT);
    if (warp == 9) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem, 512);
    }
}

// Short portions of many heads take the warp-level form, four CTAs of which share a multiprocessor (a CTA here takes 5 us beside its
// chunks): 16 tokens, 1024 heads 43 us here, 41 there; 20 tokens, 8192 heads 347 and 303; 16 tokens, 256 heads 13 and 16; 65 tokens, 1024
// heads 44 and 65.
bool ssd_scan_tc_ok(const SsmScanParams& p) {
    return (p.S > 64 || (long long)p.B * p.H <= 4 * sm_count()) && p.P == ST_P && p.N == ST_N && p.xbc_ld % 8 == 0 && p.y_ld % 8 == 0 &&
           ((reinterpret_cast<uintptr_t>(p.xbc) | reinterpret_cast<uintptr_t>(p.y)) & 15) == 0 && (long long)p.B * p.H <= 0x7fffffff;
}

int ssd_scan_tc(const SsmScanParams& p, int* error_word, cudaStream_t st) {
    const char* what = "bn_ssm_scan_checked";
    static thread_local int configured_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (configured_dev != dev) {
        cudaError_t e = cudaFuncSetAttribute(ssd_scan_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ST_SMEM);
        if (e != cudaSuccess) return fail(BN_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
        configured_dev = dev;
    }
    // (column, token, sequence); one box = 64 columns of 128 tokens, zeros (or nothing written) beyond the sequence
    CUtensorMap map, map_y;
    const uint64_t dims[3] = {(uint64_t)(p.H * p.P + 2 * p.G * p.N), (uint64_t)p.S, (uint64_t)p.B}, dims_y[3] = {(uint64_t)(p.H * p.P), (uint64_t)p.S, (uint64_t)p.B};
    const uint64_t strides[2] = {(uint64_t)p.xbc_ld * 2, (uint64_t)p.xbc_ld * 2 * p.S}, strides_y[2] = {(uint64_t)p.y_ld * 2, (uint64_t)p.y_ld * 2 * p.S};
    const uint32_t box[3] = {64, ST_Q, 1};
    if (int rc = make_tensor_map(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, p.xbc, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B)) return rc;
    if (int rc = make_tensor_map(&map_y, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, p.y, dims_y, strides_y, box, CU_TENSOR_MAP_SWIZZLE_128B)) return rc;
    launch_dependent(ssd_scan_tc_kernel, (unsigned)(p.B * p.H), ST_THREADS, ST_SMEM, st, map, map_y, StParams{p, error_word});
    return launch_status(what);
}

}  // namespace bn
