// Attention of a prompt portion (bn_attn_window: a sliding window and a rotated key part shared by the heads;
// bn_attn_chunked: grouped-query heads, chunks of positions, unit-RMS queries, a gate on the result) for any sizes, in fp32
// and in bf16, and the choice of the tensor-core form (attn_portion_sm100.cu).
#include <type_traits>

#include "attn_portion.cuh"
#include "common.cuh"
#include "hybrid.cuh"

namespace bn {

// ---------------------------------------------------------------------------------------------------------------
// One-token attention over cached keys, and portions of very wide heads: a warp per (query row, head); 32 keys at a time, a
// lane per key for the scores, then a lane per value column.  Scores, weights and sums in fp32.
// ---------------------------------------------------------------------------------------------------------------
constexpr int AW_WARPS = 4, AW_MAXV = 16;      // vdim <= 512

template <typename T>
__global__ void __launch_bounds__(AW_WARPS * 32)
attn_any_kernel(const AttnPortionParams p) {
    extern __shared__ float q_smem[];
    ptx::grid_dependency_wait();
    ptx::grid_launch_dependents();
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int E = p.dim + p.rot;
    float* qs = q_smem + warp * E;
    const long long n = (long long)p.B * p.S * p.H;
    for (long long item = (long long)blockIdx.x * AW_WARPS + warp; item < n; item += (long long)gridDim.x * AW_WARPS) {
        const int h = (int)(item % p.H);
        const long long row = item / p.H;
        const int b = (int)(row / p.S), s = (int)(row - (long long)b * p.S);
        const T* q = static_cast<const T*>(p.q) + row * p.q_ld + h * E;
        __syncwarp();
        float ss = 0.f;
        for (int e = lane; e < E; e += 32) { qs[e] = to_f(q[e]); ss = fmaf(qs[e], qs[e], ss); }
        __syncwarp();
        float scale = p.scale;
        if (p.rms_dim) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            scale *= rsqrtf(ss / (float)p.rms_dim + p.rms_eps);
        }
        const int g = h / (p.H / p.kv_heads), block = p.seq_ids ? p.seq_ids[b] : b;
        const int last = p.positions ? p.positions[b] % p.span : p.n_old + s, first = max(0, mask_oldest(p.mask, p.span, last));
        if (p.positions && last >= p.rows_per_seq) {       // the cache has no room for this token
            for (int v = lane; v < p.vdim; v += 32)
                static_cast<T*>(p.out)[row * p.out_ld + h * p.vdim + v] = from_f<T>(__int_as_float(0x7fc00000));
            continue;
        }
        const T* kseq = static_cast<const T*>(p.k) + block * p.k_seq + g * p.k_head;
        const T* vseq = static_cast<const T*>(p.v) + block * p.v_seq + g * p.v_head;
        const T* kr_seq = static_cast<const T*>(p.krot) + (int64_t)b * p.rows_per_seq * p.krot_ld;
        float m = -INFINITY, l = 0.f, acc[AW_MAXV];
#pragma unroll
        for (int v = 0; v < AW_MAXV; ++v) acc[v] = 0.f;
        for (int k0 = first; k0 <= last; k0 += 32) {
            const int k = k0 + lane;
            float sc = -INFINITY;
            if (k <= last) {
                const T* kn = kseq + k * p.k_ld;
                const T* kr = kr_seq + k * p.krot_ld;
                float d = 0.f;
                for (int e = 0; e < p.dim; ++e) d = fmaf(qs[e], to_f(kn[e]), d);
                for (int e = 0; e < p.rot; ++e) d = fmaf(qs[p.dim + e], to_f(kr[e]), d);
                sc = d * scale;
            }
            float mx = sc;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            const float m_new = fmaxf(m, mx);
            const float shrink = expf(m - m_new);      // 0 at the first keys (m = -inf)
            const float w = expf(sc - m_new);
            float sum = w;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            l = l * shrink + sum;
            m = m_new;
#pragma unroll
            for (int v = 0; v < AW_MAXV; ++v) acc[v] *= shrink;
            const int nk = min(32, last - k0 + 1);
            for (int j = 0; j < nk; ++j) {
                const float wj = __shfl_sync(0xffffffffu, w, j);
                const T* vr = vseq + (k0 + j) * p.v_ld;
#pragma unroll
                for (int v = 0; v < AW_MAXV; ++v)
                    if (v * 32 + lane < p.vdim) acc[v] = fmaf(wj, to_f(vr[v * 32 + lane]), acc[v]);
            }
        }
        T* out = static_cast<T*>(p.out) + row * p.out_ld + h * p.vdim;
#pragma unroll
        for (int v = 0; v < AW_MAXV; ++v)
            if (v * 32 + lane < p.vdim) {
                float o = acc[v] / l;
                if (p.gate) o *= sigmoid_exact(to_f(static_cast<const T*>(p.gate)[row * p.gate_ld + h * p.vdim + v * 32 + lane]));
                out[v * 32 + lane] = from_f<T>(o);
            }
        if (h == p.H - 1)                                   // the padding columns behind the last head
            for (int i = p.H * p.vdim + lane; i < p.out_ld; i += 32)
                static_cast<T*>(p.out)[row * p.out_ld + i] = from_f<T>(0.f);
    }
}

// ---------------------------------------------------------------------------------------------------------------
// Portion attention in tiles, any head sizes: what attn_any_kernel computes, with keys and queries in shared memory.  A CTA
// owns AT_ROWS rows of one sequence and key head, a row = (query position, one of the query heads that share the key head),
// positions slowest.  64 keys at a time: thread = (key, group of AT_RPT rows) for the scores, whose columns come in pieces of
// 64; a warp per row for the running maximum and sum; thread = (value column mod 64, group of rows) for the result, which
// reads a value from global memory once for AT_RPT rows.  fp32 throughout, a score is one FMA chain over its columns.
// The warp-per-row kernel reads every key for every row, 32 rows of a matrix at a time: 32 heads over 4 x 64 columns, 4 x 200
// tokens, 873 us; this one 129 us.
// A tile of keys where the mask of some row cuts leaves the masked (row, key) pairs out of the result, as that kernel does: their
// weight is no zero to multiply by, or a value that is not finite would reach rows that do not see it.
// ---------------------------------------------------------------------------------------------------------------
constexpr int AT_KEYS = 64, AT_RPT = 8, AT_ROWS = 32, AT_THREADS = AT_KEYS * AT_ROWS / AT_RPT, AT_E = 64, AT_KLD = AT_E + 4;

// VB: value columns in blocks of 64.
template <typename T, int VB>
__global__ void __launch_bounds__(AT_THREADS, 1)
attn_tiled_kernel(const AttnPortionParams p) {
    extern __shared__ __align__(16) float at_smem[];
    __shared__ __align__(16) float Ks[AT_KEYS * AT_KLD];
    __shared__ __align__(16) float Ps[AT_ROWS][AT_KEYS + 4];
    __shared__ float row_m[AT_ROWS], row_l[AT_ROWS], row_shrink[AT_ROWS], row_scale[AT_ROWS];
    ptx::grid_dependency_wait();
    ptx::grid_launch_dependents();
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32, key = tid % AT_KEYS, group = tid / AT_KEYS;
    const int E = p.dim + p.rot, q_ld = (E + 3) / 4 * 4 + 4, n_rep = p.H / p.kv_heads;
    float* Qs = at_smem;                                       // [row][q_ld], zeros behind the columns
    const int tiles_per_seq = (int)(((long long)p.S * n_rep + AT_ROWS - 1) / AT_ROWS);
    const int tile = tiles_per_seq - 1 - (int)(blockIdx.x % tiles_per_seq), bg = (int)(blockIdx.x / tiles_per_seq);
    const int b = bg / p.kv_heads, g = bg % p.kv_heads, t0 = tile * AT_ROWS, n_rows = min(AT_ROWS, p.S * n_rep - t0);
    auto position = [&](int r) { return (t0 + r) / n_rep; };   // of the portion
    auto head = [&](int r) { return g * n_rep + (t0 + r) % n_rep; };

    for (int r = warp; r < AT_ROWS; r += AT_THREADS / 32) {
        float ss = 0.f;
        const T* q = static_cast<const T*>(p.q) + ((int64_t)b * p.S + position(r)) * p.q_ld + head(r) * E;
        for (int e = lane; e < q_ld; e += 32) {
            const float v = r < n_rows && e < E ? to_f(q[e]) : 0.f;
            Qs[r * q_ld + e] = v;
            ss = fmaf(v, v, ss);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if (lane == 0) {
            row_scale[r] = p.rms_dim ? p.scale * rsqrtf(ss / (float)p.rms_dim + p.rms_eps) : p.scale;
            row_m[r] = -INFINITY;
            row_l[r] = 0.f;
        }
    }
    const int first = max(0, mask_oldest(p.mask, p.span, p.n_old + position(0))), last = p.n_old + position(n_rows - 1);
    const T* kseq = static_cast<const T*>(p.k) + b * p.k_seq + g * p.k_head;
    const T* vseq = static_cast<const T*>(p.v) + b * p.v_seq + g * p.v_head;
    const T* kr_seq = static_cast<const T*>(p.krot) + (int64_t)b * p.rows_per_seq * p.krot_ld;
    float acc[AT_RPT][VB];
#pragma unroll
    for (int r = 0; r < AT_RPT; ++r)
#pragma unroll
        for (int v = 0; v < VB; ++v) acc[r][v] = 0.f;

    for (int k0 = first; k0 <= last; k0 += AT_KEYS) {
        float s[AT_RPT];
#pragma unroll
        for (int r = 0; r < AT_RPT; ++r) s[r] = 0.f;
        for (int e0 = 0; e0 < E; e0 += AT_E) {
            __syncthreads();                                   // the piece before (and the weights) have been read
#pragma unroll 8
            for (int i = tid; i < AT_KEYS * AT_E; i += AT_THREADS) {
                const int kk = i / AT_E, e = e0 + i % AT_E, k = k0 + kk;
                Ks[kk * AT_KLD + i % AT_E] = k > last || e >= E ? 0.f : e < p.dim ? to_f(kseq[(int64_t)k * p.k_ld + e])
                                                                                  : to_f(kr_seq[(int64_t)k * p.krot_ld + e - p.dim]);
            }
            __syncthreads();
            const int n = min(AT_E, E - e0);
#pragma unroll 2
            for (int e = 0; e < n; e += 4) {                   // (a piece's last columns may be the zeros behind the row)
                const float4 k4 = *reinterpret_cast<const float4*>(Ks + key * AT_KLD + e);
#pragma unroll
                for (int r = 0; r < AT_RPT; ++r) {
                    const float4 q4 = *reinterpret_cast<const float4*>(Qs + (group * AT_RPT + r) * q_ld + e0 + e);
                    s[r] = fmaf(q4.w, k4.w, fmaf(q4.z, k4.z, fmaf(q4.y, k4.y, fmaf(q4.x, k4.x, s[r]))));
                }
            }
        }
#pragma unroll
        for (int r = 0; r < AT_RPT; ++r) {
            const int row = group * AT_RPT + r, own = p.n_old + position(row), k = k0 + key;
            const bool seen = row < n_rows && k <= own && k >= mask_oldest(p.mask, p.span, own);
            Ps[row][key] = seen ? s[r] * row_scale[row] : -INFINITY;
        }
        __syncthreads();
        // whether some row does not see some key of the tile
        const bool cut = k0 + AT_KEYS - 1 > p.n_old + position(0) || k0 < mask_oldest(p.mask, p.span, p.n_old + position(n_rows - 1));
        for (int r = warp; r < AT_ROWS; r += AT_THREADS / 32) {
            const float a = Ps[r][lane], c = Ps[r][lane + 32], m = row_m[r];
            float mx = fmaxf(a, c);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            const float m_new = fmaxf(m, mx);
            // nothing of the row seen yet: no weight, whatever the (masked) scores; a NaN score is seen and stays one
            const bool none = m_new == -INFINITY;
            const float wa = none && a == -INFINITY ? 0.f : expf(a - m_new), wc = none && c == -INFINITY ? 0.f : expf(c - m_new);
            float sum = wa + wc;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            if (cut) {                                         // a masked pair's weight: -1
                const int own = p.n_old + position(r), oldest = mask_oldest(p.mask, p.span, own), k = k0 + lane;
                Ps[r][lane] = k <= own && k >= oldest ? wa : -1.f;
                Ps[r][lane + 32] = k + 32 <= own && k + 32 >= oldest ? wc : -1.f;
            } else {
                Ps[r][lane] = wa;
                Ps[r][lane + 32] = wc;
            }
            if (lane == 0) {
                const float shrink = none ? 1.f : expf(m - m_new);
                row_shrink[r] = shrink;
                row_l[r] = row_l[r] * shrink + sum;
                row_m[r] = m_new;
            }
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < AT_RPT; ++r) {
            const float shrink = row_shrink[group * AT_RPT + r];
#pragma unroll
            for (int v = 0; v < VB; ++v) acc[r][v] *= shrink;
        }
        const int nk = min(AT_KEYS, last - k0 + 1);
        auto apply = [&](auto masked) {
            auto add = [&](float w, float v, float sum) { return decltype(masked)::value && w < 0.f ? sum : fmaf(w, v, sum); };
#pragma unroll 2
            for (int j = 0; j < nk; j += 4) {
                float val[4][VB];
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int v = 0; v < VB; ++v)
                        val[i][v] = j + i < nk && v * 64 + key < p.vdim ? to_f(vseq[(int64_t)(k0 + j + i) * p.v_ld + v * 64 + key]) : 0.f;
#pragma unroll
                for (int r = 0; r < AT_RPT; ++r) {
                    const float4 w = *reinterpret_cast<const float4*>(&Ps[group * AT_RPT + r][j]);
#pragma unroll
                    for (int v = 0; v < VB; ++v)
                        acc[r][v] = add(w.w, val[3][v], add(w.z, val[2][v], add(w.y, val[1][v], add(w.x, val[0][v], acc[r][v]))));
                }
            }
        };
        if (cut) apply(std::true_type{});
        else apply(std::false_type{});
    }
#pragma unroll
    for (int r = 0; r < AT_RPT; ++r) {
        const int row = group * AT_RPT + r;
        if (row >= n_rows) continue;
        const int64_t at = (int64_t)b * p.S + position(row);
        const int h = head(row);
        T* out = static_cast<T*>(p.out) + at * p.out_ld;
#pragma unroll
        for (int v = 0; v < VB; ++v) {
            const int c = v * 64 + key;
            if (c >= p.vdim) continue;
            float o = acc[r][v] / row_l[row];
            if (p.gate) o *= sigmoid_exact(to_f(static_cast<const T*>(p.gate)[at * p.gate_ld + h * p.vdim + c]));
            out[h * p.vdim + c] = from_f<T>(o);
        }
        if (h == p.H - 1)                                      // the padding columns behind the last head
            for (int i = p.H * p.vdim + key; i < p.out_ld; i += AT_KEYS) out[i] = from_f<T>(0.f);
    }
}

// ---------------------------------------------------------------------------------------------------------------
// The same in fp32 for rows of whole 16-byte pieces: a CTA owns 64 rows, and a thread 8 rows x 4 keys of the scores and 8 rows x 4
// columns (of each 64) of the result, 12 16-byte reads of shared memory for 128 FMAs; those reads bind (the kernel above has 9 for
// 32).  Keys come in pieces of 64 columns by cp.async, one ahead, values under the scores; maximum, sum and weights of a row stay
// with the 16 threads that have it.  Scores and results are the same chains as above.
// 32 heads over 4 x 64 columns, 4 x 200 tokens, 63 us; with 8 rows x 1 key a thread 96 us, with 8 x 4 in 128 threads (two warps a
// scheduler, which show every latency) 97 us, with the tiles of one sequence one behind the other 68 us.
// ---------------------------------------------------------------------------------------------------------------
constexpr int AP_ROWS = 64, AP_KEYS = 64, AP_THREADS = 256, AP_LD = 68;

template <int VB>
__global__ void __launch_bounds__(AP_THREADS, VB == 1 ? 3 : 2)
attn_tiles_f32_kernel(const AttnPortionParams p) {
    extern __shared__ __align__(16) float at_smem[];
    ptx::grid_dependency_wait();
    ptx::grid_launch_dependents();
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32, tx = tid % 16, ty = tid / 16;
    const int E = p.dim + p.rot, pieces = (E + 63) / 64, q_ld = pieces * 64 + 4, n_rep = p.H / p.kv_heads;
    constexpr int V_LD = VB * 64;
    float* Ks = at_smem;                                       // [64][68]
    float* Vs = Ks + AP_KEYS * AP_LD;                      // [64][V_LD]
    float* Ps = Vs + AP_KEYS * V_LD;                           // [64][68]
    float* Qs = Ps + AP_ROWS * AP_LD;                          // [64][q_ld], zeros behind the columns
    float* row_scale = Qs + AP_ROWS * q_ld;
    const int tiles_per_seq = (int)(((long long)p.S * n_rep + AP_ROWS - 1) / AP_ROWS);
    // the tiles with most keys first, of all sequences and heads: a multiprocessor then gets a long, a middle and a short one
    const int bgs = p.B * p.kv_heads, tile = tiles_per_seq - 1 - (int)(blockIdx.x / bgs), bg = (int)(blockIdx.x % bgs);
    const int b = bg / p.kv_heads, g = bg % p.kv_heads, t0 = tile * AP_ROWS, n_rows = min(AP_ROWS, p.S * n_rep - t0);
    auto position = [&](int r) { return (t0 + r) / n_rep; };   // of the portion
    auto head = [&](int r) { return g * n_rep + (t0 + r) % n_rep; };
    const int first = max(0, mask_oldest(p.mask, p.span, p.n_old + position(0))), last = p.n_old + position(n_rows - 1);
    const int key_tiles = (last - first) / AP_KEYS + 1;
    const float* kseq = static_cast<const float*>(p.k) + b * p.k_seq + g * p.k_head;
    const float* vseq = static_cast<const float*>(p.v) + b * p.v_seq + g * p.v_head;
    const float* kr_seq = static_cast<const float*>(p.krot) + (int64_t)b * p.rows_per_seq * p.krot_ld;
    const uint32_t uK = ptx::smem_u32(Ks), uV = ptx::smem_u32(Vs);

    // piece n of the keys: columns 64 (n % pieces) .. of key tile n / pieces; what lies outside becomes zero
    auto ask_keys = [&](int n) {
        if (n < key_tiles * pieces) {
            const int k0 = first + n / pieces * AP_KEYS, e0 = n % pieces * 64;
#pragma unroll
            for (int i = 0; i < AP_KEYS * 16 / AP_THREADS; ++i) {
                const int kk = ty + i * (AP_THREADS / 16), e = e0 + tx * 4, k = k0 + kk;
                const bool in = k <= last && e < E;
                const float* at = e < p.dim ? kseq + (int64_t)k * p.k_ld + e : kr_seq + (int64_t)k * p.krot_ld + e - p.dim;
                ptx::cp_async_16(uK + (kk * AP_LD + tx * 4) * 4, in ? at : kseq, in ? 16 : 0);
            }
        }
        ptx::cp_async_commit();
    };
    auto ask_values = [&](int t) {
        const int k0 = first + t * AP_KEYS;
#pragma unroll
        for (int i = 0; i < AP_KEYS * 16 / AP_THREADS; ++i) {
            const int kk = ty + i * (AP_THREADS / 16);
#pragma unroll
            for (int v = 0; v < VB; ++v) {
                const int c = v * 64 + tx * 4;
                const bool in = k0 + kk <= last && c < p.vdim;
                ptx::cp_async_16(uV + (kk * V_LD + c) * 4, in ? vseq + (int64_t)(k0 + kk) * p.v_ld + c : vseq, in ? 16 : 0);
            }
        }
        ptx::cp_async_commit();
    };
    ask_keys(0);
    for (int r = warp; r < AP_ROWS; r += AP_THREADS / 32) {
        float ss = 0.f;
        const float* q = static_cast<const float*>(p.q) + ((int64_t)b * p.S + position(r)) * p.q_ld + head(r) * E;
        for (int e = lane; e < pieces * 64; e += 32) {
            const float v = r < n_rows && e < E ? q[e] : 0.f;
            Qs[r * q_ld + e] = v;
            ss = fmaf(v, v, ss);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if (lane == 0) row_scale[r] = p.rms_dim ? p.scale * rsqrtf(ss / (float)p.rms_dim + p.rms_eps) : p.scale;
    }
    // this thread's rows: ty + 16 i
    float acc[4][VB][4], m[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.f;
#pragma unroll
        for (int v = 0; v < VB; ++v) acc[i][v][0] = acc[i][v][1] = acc[i][v][2] = acc[i][v][3] = 0.f;
    }
    for (int t = 0, n = 0; t < key_tiles; ++t) {
        const int k0 = first + t * AP_KEYS;
        float s[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f;
        for (int piece = 0; piece < pieces; ++piece, ++n) {
            ptx::cp_async_wait<0>();                           // these keys (and the values before the last piece)
            __syncthreads();
            if (piece == 0) ask_values(t);
            const float* ks = Ks + tx * AP_LD;
            const float* qs = Qs + ty * q_ld + piece * 64;
#pragma unroll 2
            for (int e = 0; e < 64; e += 4) {                  // (the last columns may be zeros on both sides)
                float4 k4[4], q4[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) k4[j] = *reinterpret_cast<const float4*>(ks + j * 16 * AP_LD + e);
#pragma unroll
                for (int i = 0; i < 4; ++i) q4[i] = *reinterpret_cast<const float4*>(qs + i * 16 * q_ld + e);
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        s[i][j] = fmaf(q4[i].w, k4[j].w, fmaf(q4[i].z, k4[j].z, fmaf(q4[i].y, k4[j].y, fmaf(q4[i].x, k4[j].x, s[i][j]))));
            }
            __syncthreads();                                   // the piece has been read
            ask_keys(n + 1);
        }
        // whether some row does not see some key of the tile
        const bool cut = k0 + AP_KEYS - 1 > p.n_old + position(0) || k0 < mask_oldest(p.mask, p.span, p.n_old + position(n_rows - 1)) || n_rows < AP_ROWS;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = ty + i * 16, own = p.n_old + position(r), oldest = mask_oldest(p.mask, p.span, own);
            const float scale = row_scale[r];
            bool seen[4];
            float mx = -INFINITY;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int k = k0 + tx + j * 16;
                seen[j] = !cut || (r < n_rows && k <= own && k >= oldest);
                s[i][j] = seen[j] ? s[i][j] * scale : -INFINITY;
                mx = fmaxf(mx, s[i][j]);
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            const float m_new = fmaxf(m[i], mx);
            // nothing of the row seen yet: no weight, whatever the (masked) scores; a NaN score is seen and stays one
            const bool none = m_new == -INFINITY;
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float w = none && s[i][j] == -INFINITY ? 0.f : expf(s[i][j] - m_new);
                sum += w;
                Ps[r * AP_LD + tx + j * 16] = seen[j] ? w : -1.f;          // a masked pair's weight: -1
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            const float shrink = none ? 1.f : expf(m[i] - m_new);
            l[i] = l[i] * shrink + sum;
            m[i] = m_new;
#pragma unroll
            for (int v = 0; v < VB; ++v)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[i][v][c] *= shrink;
        }
        ptx::cp_async_wait<1>();                               // the values; the next keys are on their way
        __syncthreads();
        const int nk = min(AP_KEYS, last - k0 + 1);
        auto apply = [&](auto masked) {
            auto add = [&](float w, float v, float sum) { return decltype(masked)::value && w < 0.f ? sum : fmaf(w, v, sum); };
#pragma unroll 2
            for (int j = 0; j < nk; j += 4) {                  // (weights beyond the last key are -1 or, uncut, there are none)
                float4 w4[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) w4[i] = *reinterpret_cast<const float4*>(Ps + (ty + i * 16) * AP_LD + j);
#pragma unroll
                for (int v = 0; v < VB; ++v) {
                    float4 x[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) x[e] = *reinterpret_cast<const float4*>(Vs + (j + e) * V_LD + v * 64 + tx * 4);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        float(&a)[4] = acc[i][v];
                        a[0] = add(w4[i].w, x[3].x, add(w4[i].z, x[2].x, add(w4[i].y, x[1].x, add(w4[i].x, x[0].x, a[0]))));
                        a[1] = add(w4[i].w, x[3].y, add(w4[i].z, x[2].y, add(w4[i].y, x[1].y, add(w4[i].x, x[0].y, a[1]))));
                        a[2] = add(w4[i].w, x[3].z, add(w4[i].z, x[2].z, add(w4[i].y, x[1].z, add(w4[i].x, x[0].z, a[2]))));
                        a[3] = add(w4[i].w, x[3].w, add(w4[i].z, x[2].w, add(w4[i].y, x[1].w, add(w4[i].x, x[0].w, a[3]))));
                    }
                }
            }
        };
        if (cut) apply(std::true_type{});
        else apply(std::false_type{});
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = ty + i * 16;
        if (r >= n_rows) continue;
        const int64_t at = (int64_t)b * p.S + position(r);
        const int h = head(r);
        float* out = static_cast<float*>(p.out) + at * p.out_ld;
#pragma unroll
        for (int v = 0; v < VB; ++v)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int col = v * 64 + tx * 4 + c;
                if (col >= p.vdim) continue;
                float o = acc[i][v][c] / l[i];
                if (p.gate) o *= sigmoid_exact(static_cast<const float*>(p.gate)[at * p.gate_ld + h * p.vdim + col]);
                out[h * p.vdim + col] = o;
            }
        if (h == p.H - 1)                                      // the padding columns behind the last head
            for (int c = p.H * p.vdim + tx; c < p.out_ld; c += 16) out[c] = 0.f;
    }
}

static size_t attn_tiles_f32_smem(const AttnPortionParams& p) {
    const int pieces = (p.dim + p.rot + 63) / 64, blocks = (p.vdim + 63) / 64;
    return (size_t)(AP_KEYS * AP_LD + AP_KEYS * blocks * 64 + AP_ROWS * (AP_LD + pieces * 64 + 4 + 1)) * sizeof(float);
}

// Whole 16-byte pieces of keys and values at 16-byte addresses, at most 128 value columns, and room for the queries
static bool attn_tiles_f32_ok(const AttnPortionParams& p) {
    const uintptr_t at = reinterpret_cast<uintptr_t>(p.k) | reinterpret_cast<uintptr_t>(p.v) | (p.rot ? reinterpret_cast<uintptr_t>(p.krot) : 0);
    return p.vdim <= 128 && (p.dim | p.rot | p.vdim) % 4 == 0 && (p.k_ld | p.v_ld | p.k_seq | p.v_seq | p.k_head | p.v_head) % 4 == 0 &&
           (p.rot == 0 || p.krot_ld % 4 == 0) && (at & 15) == 0 && attn_tiles_f32_smem(p) <= 200 * 1024;
}

template <int VB>
static int attn_tiles_f32(const AttnPortionParams& p, cudaStream_t st, const char* what) {
    const long long tiles = ((long long)p.S * (p.H / p.kv_heads) + AP_ROWS - 1) / AP_ROWS, blocks = tiles * p.B * p.kv_heads;
    if (blocks > 0x7fffffffLL) return fail(BN_ERR_UNSUPPORTED, "%s: B=%d x S=%d too large", what, p.B, p.S);
    const size_t smem = attn_tiles_f32_smem(p);
    if (int rc = allow_smem(attn_tiles_f32_kernel<VB>, smem, what)) return rc;
    launch_dependent(attn_tiles_f32_kernel<VB>, (unsigned)blocks, AP_THREADS, smem, st, p);
    return launch_status(what);
}

// ---------------------------------------------------------------------------------------------------------------
// One new fp32 token a sequence over its cached keys.  A cluster of up to eight CTAs per (sequence, key head, group of eight of
// its query heads): block j of 32 keys belongs to warp j / ranks of CTA j % ranks, so that short and long sequences both spread
// over all warps, and a key or value is read once for eight heads.  A warp has all keys and values of its block on their way
// into shared memory at once; a lane = (head, every fourth key) for the scores and weights, VC value columns of all eight
// heads for the result.  Warps keep their own maxima and meet in shared memory, CTAs in each other's (the entry has no scratch
// memory to give).
// What bounds it is latency: 1024 keys of 64 columns are one pass of a cluster's 32 warps.  The loops are unrolled no further
// than loads need: a step meets this code cold, and the same work in 2500 instructions in a row took 28 us however short the
// sequence was.  A warp per head that walks the keys by itself (attn_any_kernel) is a chain of rounds: 32 heads over 4 x 64
// columns, 4 sequences of 400 tokens, 580 us; this 13.
// ---------------------------------------------------------------------------------------------------------------
constexpr int SA_WARPS = 4, SA_HEADS = 8, SA_MAXRANKS = 8, SA_THREADS = SA_WARPS * 32;

// E, V: columns of keys and values in shared memory (64 or 128 each)
template <int E, int V>
struct SaShape {
    static constexpr int LD = E + 4;
    static constexpr int SMEM_BYTES = SA_WARPS * 32 * (LD + V) * 4;
};

template <int E, int V>
__global__ void __launch_bounds__(SA_THREADS)
attn_step_f32_kernel(const AttnPortionParams p, int ranks) {
    constexpr int LD = SaShape<E, V>::LD, VC = V / 32;
    extern __shared__ __align__(16) float sa_smem[];
    __shared__ __align__(16) float qs[SA_HEADS][LD];                           // zeros behind the columns and the heads
    __shared__ __align__(16) float ws[SA_WARPS][32][SA_HEADS], part[SA_WARPS][SA_HEADS][V], cta[SA_HEADS][V];
    __shared__ float shr[SA_WARPS][SA_HEADS], wm[SA_WARPS][SA_HEADS], wl[SA_WARPS][SA_HEADS], cm[SA_HEADS], cl[SA_HEADS], hs[SA_HEADS],
        share[SA_MAXRANKS][SA_HEADS];
    ptx::grid_dependency_wait();
    ptx::grid_launch_dependents();
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32, rank = (int)ptx::cluster_rank();
    const int n_rep = p.H / p.kv_heads, hgs = (n_rep + SA_HEADS - 1) / SA_HEADS, item = blockIdx.x / ranks;
    const int hg = item % hgs, g = item / hgs % p.kv_heads, b = item / (hgs * p.kv_heads);
    const int h0 = g * n_rep + hg * SA_HEADS, heads = min(SA_HEADS, n_rep - hg * SA_HEADS);
    const int block = p.seq_ids ? p.seq_ids[b] : b, last = p.positions[b] % p.span, first = max(0, mask_oldest(p.mask, p.span, last));
    const bool room = last < p.rows_per_seq;                                   // else the cache has no room for this token
    const float* kseq = static_cast<const float*>(p.k) + block * p.k_seq + g * p.k_head;
    const float* vseq = static_cast<const float*>(p.v) + block * p.v_seq + g * p.v_head;
    float* Ks = sa_smem + warp * 32 * (LD + V);
    float* Vs = Ks + 32 * LD;
    auto fetch = [&](int k0) {                                                 // two groups: keys, values
#pragma unroll 4
        for (int i = lane; i < 32 * (E / 4); i += 32) {
            const int k = i / (E / 4), e = i % (E / 4) * 4;
            const bool in = k0 + k <= last && e < p.dim;
            ptx::cp_async_16(ptx::smem_u32(Ks + k * LD + e), kseq + (in ? (k0 + k) * p.k_ld + e : 0), in ? 16 : 0);
        }
        ptx::cp_async_commit();
#pragma unroll 4
        for (int i = lane; i < 32 * (V / 4); i += 32) {
            const int k = i / (V / 4), c = i % (V / 4) * 4;
            const bool in = k0 + k <= last && c < p.vdim;
            ptx::cp_async_16(ptx::smem_u32(Vs + k * V + c), vseq + (in ? (k0 + k) * p.v_ld + c : 0), in ? 16 : 0);
        }
        ptx::cp_async_commit();
    };
    int k0 = room ? first + (warp * ranks + rank) * 32 : last + 1;
    if (k0 <= last) fetch(k0);
#pragma unroll 1
    for (int h = warp; h < SA_HEADS; h += SA_WARPS) {
        const float* q = static_cast<const float*>(p.q) + b * p.q_ld + (int64_t)(h0 + h) * p.dim;
        float ss = 0.f;
#pragma unroll
        for (int e = lane; e < E; e += 32) {
            const float x = h < heads && e < p.dim ? q[e] : 0.f;
            qs[h][e] = x;
            ss = fmaf(x, x, ss);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if (lane == 0) hs[h] = p.rms_dim ? p.scale * rsqrtf(ss / (float)p.rms_dim + p.rms_eps) : p.scale;
    }
    __syncthreads();
    const int hw = lane / 4, kw = lane % 4, c0 = lane * VC;
    float m = -INFINITY, l = 0.f, acc[SA_HEADS][VC];
#pragma unroll
    for (int h = 0; h < SA_HEADS; ++h)
#pragma unroll
        for (int c = 0; c < VC; ++c) acc[h][c] = 0.f;
#pragma unroll 1
    for (; k0 <= last; ) {
        ptx::cp_async_wait<1>();
        __syncwarp();
        float mx = m;
#pragma unroll 1
        for (int i = 0; i < 8; i += 2) {                                       // two keys a lane at a time
            float d0 = 0.f, d1 = 0.f;
#pragma unroll 8
            for (int e = 0; e < E; e += 4) {
                float qv[4], ka[4], kb[4];
                load4(&qs[hw][e], qv);
                load4(Ks + (i * 4 + kw) * LD + e, ka);
                load4(Ks + (i * 4 + 4 + kw) * LD + e, kb);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    d0 = fmaf(qv[j], ka[j], d0);
                    d1 = fmaf(qv[j], kb[j], d1);
                }
            }
            d0 = k0 + i * 4 + kw <= last ? d0 * hs[hw] : -INFINITY;
            d1 = k0 + i * 4 + 4 + kw <= last ? d1 * hs[hw] : -INFINITY;
            ws[warp][i * 4 + kw][hw] = d0;
            ws[warp][i * 4 + 4 + kw][hw] = d1;
            mx = fmaxf(mx, fmaxf(d0, d1));
        }
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        const float base = mx == -INFINITY ? 0.f : mx, shrink = expf(m - base);          // 0 at the first keys (m = -inf)
        float sum = 0.f;
#pragma unroll 2
        for (int i = 0; i < 8; ++i) {
            const float w = expf(ws[warp][i * 4 + kw][hw] - base);
            sum += w;
            ws[warp][i * 4 + kw][hw] = w;
        }
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        l = l * shrink + sum;
        m = mx;
        if (kw == 0) shr[warp][hw] = shrink;
        ptx::cp_async_wait<0>();
        __syncwarp();
#pragma unroll
        for (int h = 0; h < SA_HEADS; ++h)
#pragma unroll
            for (int c = 0; c < VC; ++c) acc[h][c] *= shr[warp][h];
        const int nk = min(32, last - k0 + 1);
#pragma unroll 4
        for (int j = 0; j < nk; ++j) {
            float vx[VC], w8[SA_HEADS];
            if (VC == 4) load4(Vs + j * V + c0, *reinterpret_cast<float(*)[4]>(vx));
            else { const float2 t = *reinterpret_cast<const float2*>(Vs + j * V + c0); vx[0] = t.x; vx[1] = t.y; }
            load4(&ws[warp][j][0], *reinterpret_cast<float(*)[4]>(w8));
            load4(&ws[warp][j][4], *reinterpret_cast<float(*)[4]>(w8 + 4));
#pragma unroll
            for (int h = 0; h < SA_HEADS; ++h)
#pragma unroll
                for (int c = 0; c < VC; ++c) acc[h][c] = fmaf(w8[h], vx[c], acc[h][c]);
        }
        __syncwarp();
        k0 += 32 * SA_WARPS * ranks;
        if (k0 <= last) fetch(k0);
    }
#pragma unroll
    for (int h = 0; h < SA_HEADS; ++h)
#pragma unroll
        for (int c = 0; c < VC; ++c) part[warp][h][c0 + c] = acc[h][c];
    if (kw == 0) { wm[warp][hw] = m; wl[warp][hw] = l; }
    __syncthreads();
    if (tid < SA_HEADS) {                                                      // the CTA's warps
        float top = -INFINITY, sum = 0.f;
        for (int w = 0; w < SA_WARPS; ++w) top = fmaxf(top, wm[w][tid]);
        const float base = top == -INFINITY ? 0.f : top;
#pragma unroll 1
        for (int w = 0; w < SA_WARPS; ++w) {
            const float f = expf(wm[w][tid] - base);
            shr[w][tid] = f;
            sum = fmaf(wl[w][tid], f, sum);
        }
        cm[tid] = top;
        cl[tid] = sum;
    }
    __syncthreads();
    for (int i = tid; i < SA_HEADS * V; i += SA_THREADS) {
        const int h = i / V, c = i % V;
        float o = 0.f;
#pragma unroll
        for (int w = 0; w < SA_WARPS; ++w) o = fmaf(part[w][h][c], shr[w][h], o);
        cta[h][c] = o;
    }
    ptx::cluster_sync();
    if (tid < SA_HEADS) {                                                      // the cluster's CTAs
        float ms[SA_MAXRANKS], ls[SA_MAXRANKS], top = -INFINITY, sum = 0.f;
#pragma unroll
        for (int r = 0; r < SA_MAXRANKS; ++r) {
            ms[r] = r < ranks ? ptx::ld_cluster(ptx::in_rank(ptx::smem_u32(&cm[tid]), r)) : -INFINITY;
            ls[r] = r < ranks ? ptx::ld_cluster(ptx::in_rank(ptx::smem_u32(&cl[tid]), r)) : 0.f;
        }
#pragma unroll
        for (int r = 0; r < SA_MAXRANKS; ++r) top = fmaxf(top, ms[r]);
        const float base = top == -INFINITY ? 0.f : top;
#pragma unroll
        for (int r = 0; r < SA_MAXRANKS; ++r) {
            ms[r] = expf(ms[r] - base);
            sum = fmaf(ls[r], ms[r], sum);
        }
#pragma unroll
        for (int r = 0; r < SA_MAXRANKS; ++r) share[r][tid] = ms[r] / sum;
    }
    __syncthreads();
    for (int i = rank * SA_THREADS + tid; i < heads * p.vdim; i += ranks * SA_THREADS) {
        const int h = i / p.vdim, c = i % p.vdim;
        float part_of[SA_MAXRANKS], o = 0.f;
#pragma unroll
        for (int r = 0; r < SA_MAXRANKS; ++r) part_of[r] = r < ranks ? ptx::ld_cluster(ptx::in_rank(ptx::smem_u32(&cta[h][c]), r)) : 0.f;
#pragma unroll
        for (int r = 0; r < SA_MAXRANKS; ++r) o = fmaf(part_of[r], share[r][h], o);
        const int at = (h0 + h) * p.vdim + c;
        if (p.gate) o *= sigmoid_exact(static_cast<const float*>(p.gate)[b * p.gate_ld + at]);
        static_cast<float*>(p.out)[b * p.out_ld + at] = room ? o : __int_as_float(0x7fc00000);
    }
    if (room && rank == 0 && h0 + heads == p.H)                                // the padding columns behind the last head
        for (int64_t i = (int64_t)p.H * p.vdim + tid; i < p.out_ld; i += SA_THREADS) static_cast<float*>(p.out)[b * p.out_ld + i] = 0.f;
    ptx::cluster_sync();                                                       // nobody leaves while its sums are being read
}

// Whole 16-byte pieces of keys and values at 16-byte addresses, at most 128 columns of each, keys of their own for each head
static bool attn_step_f32_ok(const AttnPortionParams& p) {
    return p.positions && p.S == 1 && p.rot == 0 && p.dim <= 128 && p.vdim <= 128 && (p.dim | p.vdim) % 4 == 0 &&
           (p.k_ld | p.v_ld | p.k_seq | p.v_seq | p.k_head | p.v_head) % 4 == 0 &&
           ((reinterpret_cast<uintptr_t>(p.k) | reinterpret_cast<uintptr_t>(p.v)) & 15) == 0;
}

static int attn_step_f32(const AttnPortionParams& p, cudaStream_t st, const char* what) {
    const int n_rep = p.H / p.kv_heads;
    const long long items = (long long)p.B * p.kv_heads * ((n_rep + SA_HEADS - 1) / SA_HEADS), keys = p.span < p.rows_per_seq ? p.span : p.rows_per_seq;
    // as many ranks as the longest sequence has passes of a CTA's warps for, while about two CTAs a multiprocessor hold them all
    // (one where both heads are wider than 64)
    int ranks = SA_MAXRANKS;
    while (ranks > 1 && (items * ranks > 2LL * sm_count() || (ranks / 2) * 32LL * SA_WARPS >= keys)) ranks /= 2;
    if (items * ranks > 0x7fffffffLL) return fail(BN_ERR_UNSUPPORTED, "%s: B=%d too large", what, p.B);
    auto run = [&](auto kernel, size_t smem) {                                 // always the same for a kernel
        if (int rc = allow_smem(kernel, smem, what, smem)) return rc;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(items * ranks));
        cfg.blockDim = dim3(SA_THREADS);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)ranks;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 2;
        const cudaError_t e = launch_config(cfg, 1, kernel, p, ranks);
        if (e == cudaSuccess) return launch_status(what);
        (void)cudaGetLastError();
        return fail(BN_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
    };
    if (p.dim <= 64 && p.vdim <= 64) return run(attn_step_f32_kernel<64, 64>, SaShape<64, 64>::SMEM_BYTES);
    if (p.dim <= 64) return run(attn_step_f32_kernel<64, 128>, SaShape<64, 128>::SMEM_BYTES);
    if (p.vdim <= 64) return run(attn_step_f32_kernel<128, 64>, SaShape<128, 64>::SMEM_BYTES);
    return run(attn_step_f32_kernel<128, 128>, SaShape<128, 128>::SMEM_BYTES);
}

template <typename T>
static int attn_tiled(const AttnPortionParams& p, cudaStream_t st, const char* what) {
    const size_t smem = (size_t)AT_ROWS * ((p.dim + p.rot + 3) / 4 * 4 + 4) * sizeof(float);
    const long long tiles = ((long long)p.S * (p.H / p.kv_heads) + AT_ROWS - 1) / AT_ROWS, blocks = tiles * p.B * p.kv_heads;
    if (blocks > 0x7fffffffLL) return fail(BN_ERR_UNSUPPORTED, "%s: B=%d x S=%d too large", what, p.B, p.S);
    auto run = [&](auto kernel) {
        if (int rc = allow_smem(kernel, smem + 27 * 1024, what)) return rc;      // the kernel's own arrays count, too
        launch_dependent(kernel, (unsigned)blocks, AT_THREADS, smem, st, p);
        return launch_status(what);
    };
    if (p.vdim <= 64) return run(attn_tiled_kernel<T, 1>);
    if (p.vdim <= 128) return run(attn_tiled_kernel<T, 2>);
    return run(attn_tiled_kernel<T, 4>);
}

int attn_any(const AttnPortionParams& p, int dtype, cudaStream_t st, const char* what) {
    // Portions go through tiles where the rows' queries and the values' columns fit, fp32 rows of one token over a cache through a
    // cluster per key head; other one-token rows and wider heads take a warp per row.
    if (dtype == 0 && !p.positions && attn_tiles_f32_ok(p)) return p.vdim <= 64 ? attn_tiles_f32<1>(p, st, what) : attn_tiles_f32<2>(p, st, what);
    if (dtype == 0 && attn_step_f32_ok(p)) return attn_step_f32(p, st, what);
    if (!p.positions && p.vdim <= 256 && p.dim + p.rot <= 1024)
        return dtype == 0 ? attn_tiled<float>(p, st, what) : attn_tiled<__nv_bfloat16>(p, st, what);
    if (p.vdim > AW_MAXV * 32) return fail(BN_ERR_UNSUPPORTED, "%s: vdim=%d (at most %d)", what, p.vdim, AW_MAXV * 32);
    const size_t smem = (size_t)AW_WARPS * (p.dim + p.rot) * sizeof(float);
    const long long blocks = ((long long)p.B * p.S * p.H + AW_WARPS - 1) / AW_WARPS, cap = (long long)sm_count() * 64;
    const unsigned grid = (unsigned)(blocks < cap ? blocks : cap);
    if (dtype == 0) {
        if (int rc = allow_smem(attn_any_kernel<float>, smem, what)) return rc;
        launch_dependent(attn_any_kernel<float>, grid, AW_WARPS * 32, smem, st, p);
    } else {
        if (int rc = allow_smem(attn_any_kernel<__nv_bfloat16>, smem, what)) return rc;
        launch_dependent(attn_any_kernel<__nv_bfloat16>, grid, AW_WARPS * 32, smem, st, p);
    }
    return launch_status(what);
}

}  // namespace bn

using namespace bn;

extern "C" int bn_attn_window(const void* q, int64_t q_ld, const void* k, const void* v, int64_t kv_ld, const void* krot,
                              int64_t krot_ld, void* out, int64_t out_ld, int B, int S, int n_old, int rows_per_seq, int H,
                              int dim, int rot, int vdim, int window, float scale, int* error_word, int dtype,
                              bn_stream_t stream) {
    const char* what = "bn_attn_window";
    if (!q || !k || !v || !krot || !out) return fail(BN_ERR_INVALID_ARG, "%s: null pointer", what);
    if (B < 0 || S < 0 || n_old < 0 || n_old + S > rows_per_seq || H <= 0 || dim <= 0 || rot < 0 || vdim <= 0 || window <= 0 || (dtype & ~1))
        return fail(BN_ERR_INVALID_ARG, "%s: bad shape B=%d S=%d n_old=%d H=%d dim=%d rot=%d vdim=%d window=%d", what, B, S, n_old,
                    H, dim, rot, vdim, window);
    if (int rc = require_sm100()) return rc;
    if (B == 0 || S == 0) return BN_OK;
    AttnPortionParams p{};
    p.q = q; p.k = k; p.v = v; p.krot = krot; p.out = out;
    p.q_ld = q_ld; p.k_ld = p.v_ld = kv_ld; p.krot_ld = krot_ld; p.out_ld = out_ld;
    p.k_head = dim; p.v_head = vdim; p.k_seq = p.v_seq = rows_per_seq * kv_ld;
    p.B = B; p.S = S; p.n_old = n_old; p.rows_per_seq = rows_per_seq; p.H = p.kv_heads = H; p.dim = dim; p.rot = rot; p.vdim = vdim;
    p.mask = MASK_WINDOW; p.span = window; p.scale = scale; p.error_word = error_word;
    if (dtype == 1 && attn_portion_sm100_ok(p)) return attn_portion_sm100(p, as_stream(stream));
    return attn_any(p, dtype, as_stream(stream), what);
}

extern "C" int bn_attn_chunked(const void* q, int64_t q_ld, const void* k, int64_t k_ld, const void* v, int64_t v_ld,
                               const void* gate, int64_t gate_ld, void* out, int64_t out_ld, int B, int S, int n_old,
                               int rows_per_seq, int H, int kv_heads, int dim, int vdim, int chunk, int rms_dim, float rms_eps,
                               float scale, float score_bound, int* error_word, int dtype, bn_stream_t stream) {
    const char* what = "bn_attn_chunked";
    if (!q || !k || !v || !out) return fail(BN_ERR_INVALID_ARG, "%s: null pointer", what);
    if (B < 0 || S < 0 || n_old < 0 || n_old >= chunk || n_old + S > rows_per_seq || H <= 0 || kv_heads <= 0 || H % kv_heads || dim <= 0 ||
        vdim <= 0 || rms_dim < 0 || rms_dim > dim || (dtype & ~1))
        return fail(BN_ERR_INVALID_ARG, "%s: bad shape B=%d S=%d n_old=%d H=%d kv_heads=%d dim=%d vdim=%d chunk=%d", what, B, S, n_old, H,
                    kv_heads, dim, vdim, chunk);
    if (int rc = require_sm100()) return rc;
    if (B == 0 || S == 0) return BN_OK;
    AttnPortionParams p{};
    p.q = q; p.k = k; p.v = v; p.gate = gate; p.out = out;
    p.q_ld = q_ld; p.k_ld = k_ld; p.v_ld = v_ld; p.gate_ld = gate_ld; p.out_ld = out_ld;
    p.k_head = dim; p.v_head = vdim; p.k_seq = rows_per_seq * k_ld; p.v_seq = rows_per_seq * v_ld;
    p.B = B; p.S = S; p.n_old = n_old; p.rows_per_seq = rows_per_seq; p.H = H; p.kv_heads = kv_heads; p.dim = dim; p.vdim = vdim;
    p.mask = MASK_CHUNK; p.span = chunk; p.rms_dim = rms_dim; p.rms_eps = rms_eps; p.scale = scale; p.score_bound = score_bound;
    p.error_word = error_word;
    if (dtype == 1 && attn_portion_sm100_ok(p)) return attn_portion_sm100(p, as_stream(stream));
    return attn_any(p, dtype, as_stream(stream), what);
}
