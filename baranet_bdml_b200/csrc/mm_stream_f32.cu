// fp32 C (M,N) = act(A (M,K) W (N,K)^T + bias) for few rows: a stream of the weight through the chip.
//
// A chain of FMAs per output, which bn_mm_f32 keeps, takes K links of 4 cycles however few the rows are (2048: 4 us, and 20 - 30 us
// as tiles of 8 x 32 read their operands); here K is spread over lanes and warps and a product costs what its weight costs to read,
// up to about 16 rows, where the FMAs (one per weight and row) come to weigh as much.
// A warp owns R rows of W and a slice of K: a lane loads four k of each of them and of MM rows of A, one round of 128 k ahead of its
// use, and has R MM sums, which the lanes add up by halves (R MM shuffles where one butterfly a sum would take 5 R MM).  A block is
// four warps: WR groups of R rows, 4 / WR slices of K, added up through shared memory in order.  What is asked for in L2 before the
// wait is weights alone, as in gemm_skinny.
// A lane's sum has K / 512 to K / 128 terms of four products (more than 8 rows: four times as many links, so that FMAs alone are
// left), then pairs are added: error against 64 bits (2-norm) at most that of the sums of bn_mm_f32_sums.
// More than 16 rows go 16 at a time, the weight then coming from L2.
#include "common.cuh"
#include "hybrid.cuh"
#include "ptx.cuh"

namespace bn {

constexpr int MW_WARPS = 4, MW_ROUND = 128;

struct StreamParams {
    const float *a, *w, *bias;
    float* c;
    int64_t a_ld, w_ld, c_ld;
    int M, N, K, act, wr;
};

// Lanes add up N sums each: of two lanes O apart one goes on with the first half of them, the other with the second
template <int N, int O>
__device__ __forceinline__ void add_lanes(float* v, int lane, int& at) {
    if constexpr (O > 0) {
        if constexpr (N > 1) {
            const bool upper = lane & O;
#pragma unroll
            for (int i = 0; i < N / 2; ++i) {
                const float send = upper ? v[i] : v[i + N / 2], keep = upper ? v[i + N / 2] : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, send, O);
            }
            at += upper ? N / 2 : 0;
            add_lanes<N / 2, O / 2>(v, lane, at);
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], O);
            add_lanes<1, O / 2>(v, lane, at);
        }
    }
}

template <int R, int MM>
__global__ void __launch_bounds__(MW_WARPS * 32, 2)
mm_stream_f32_kernel(const StreamParams p) {
    constexpr int SUMS = R * MM;
    __shared__ float part[MW_WARPS][SUMS];
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, wr = warp % p.wr, wk = warp / p.wr, slices = MW_WARPS / p.wr;
    const int n0 = (blockIdx.x * p.wr + wr) * R, m0 = blockIdx.y * MM, rounds = (p.K + MW_ROUND - 1) / MW_ROUND;
    const int first = rounds * wk / slices, last = rounds * (wk + 1) / slices;
    const bool some = n0 < p.N;                                // N is a multiple of R
    const float* w = p.w + (some ? n0 : 0) * p.w_ld + lane * 4;
    const float* a = p.a + m0 * p.a_ld + lane * 4;
    if (some && lane % 8 == 0)
        for (int i = first; i < last; ++i)
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (i * MW_ROUND + lane * 4 < p.K) ptx::prefetch_l2(w + r * p.w_ld + i * MW_ROUND);
    ptx::grid_dependency_wait();
    ptx::grid_launch_dependents();
    float acc[SUMS];                                           // [row of A][row of W]
#pragma unroll
    for (int i = 0; i < SUMS; ++i) acc[i] = 0.f;
    // rows of A, which L1 and L2 hold, are asked for CH at a time, ahead of the rows before
    constexpr int CH = MM < 4 ? MM : 4, CHUNKS = MM / CH;
    float4 fw[2][R], fa[2][CH];
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    auto inside = [&](int i) { return some && i < last && i * MW_ROUND + lane * 4 < p.K; };
    auto load_w = [&](float4 (&t)[R], int i) {
        const bool in = inside(i);
#pragma unroll
        for (int r = 0; r < R; ++r) t[r] = in ? __ldcs(reinterpret_cast<const float4*>(w + r * p.w_ld + i * MW_ROUND)) : zero;
    };
    auto load_a = [&](float4 (&t)[CH], int i, int c) {
        const bool in = inside(i);
#pragma unroll
        for (int m = 0; m < CH; ++m)
            t[m] = in && m0 + c * CH + m < p.M ? *reinterpret_cast<const float4*>(a + (c * CH + m) * p.a_ld + i * MW_ROUND) : zero;
    };
    auto round = [&](int i, const float4 (&y)[R], int parity) {
#pragma unroll
        for (int c = 0; c < CHUNKS; ++c) {
            const int now = (parity * CHUNKS + c) & 1;
            if (c + 1 < CHUNKS) load_a(fa[now ^ 1], i, c + 1);
            else load_a(fa[now ^ 1], i + 1, 0);
#pragma unroll
            for (int m = 0; m < CH; ++m)
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    float& s = acc[(c * CH + m) * R + r];
                    const float4 x = fa[now][m];
                    if (MM <= 8) s += fmaf(x.w, y[r].w, fmaf(x.z, y[r].z, fmaf(x.y, y[r].y, x.x * y[r].x)));
                    else s = fmaf(x.w, y[r].w, fmaf(x.z, y[r].z, fmaf(x.y, y[r].y, fmaf(x.x, y[r].x, s))));
                }
        }
    };
    load_w(fw[0], first);
    load_a(fa[0], first, 0);
    for (int i = first; i < last; i += 2) {                    // (beyond the slice: zeros)
        load_w(fw[1], i + 1);
        round(i, fw[0], 0);
        load_w(fw[0], i + 2);
        round(i + 1, fw[1], 1);
    }
    int at = 0;                                                // the first of the sums that this lane is left with
    add_lanes<SUMS, 16>(acc, lane, at);
    constexpr int LEFT = SUMS > 32 ? SUMS / 32 : 1;
#pragma unroll
    for (int i = 0; i < LEFT; ++i) part[warp][at + i] = acc[i];          // (fewer sums than lanes: some write the same one)
    __syncthreads();
    for (int e = threadIdx.x; e < p.wr * SUMS; e += MW_WARPS * 32) {
        const int g = e / SUMS, i = e % SUMS, m = m0 + i / R, n = (blockIdx.x * p.wr + g) * R + i % R;
        if (m >= p.M || n >= p.N) continue;
        float s = part[g][i];
        for (int k = 1; k < slices; ++k) s += part[k * p.wr + g][i];
        if (p.bias) s += p.bias[n];
        p.c[m * p.c_ld + n] = activation_exact(p.act, s);
    }
}

// As many groups of R rows to a block (they share the reads of A) as leave four blocks for every multiprocessor
static int stream_groups(int N, int R) {
    int wr = MW_WARPS;
    while (wr > 1 && N / (R * wr) < 4 * sm_count()) wr /= 2;
    return wr;
}

// The time in us, roughly: a start, what a round of blocks takes beside its loads, and the weight at 5.5, 4.2 and 2.8 TB/s (the FMAs
// of 8 and 16 rows, and their reading, beside it).  us measured, with the forms there are besides (chains, sums, parts):
// 4 rows 2048 -> 7424 14.0 (35.5), 7424 -> 2048 15.4 (110.7), 2048 -> 32000 51.5 (86.3), 256 -> 2048 2.7 (4.1);
// 8 rows 20.1 (35.6), 16.9 (111.1), 73.4 (86.4), 2.7 (4.1); 16 rows 28.1 (37.1), 28.9 (109.7), 104.3 (99.7), 4.9 (4.4);
// 32 rows 50.4 (36.0), 54.9 (109.6), 201 (116), 9.2 (5.3), and 2048 -> 2048 18.3 (31.6), 2048 -> 256 3.7 (22.4).
float mm_stream_estimate(int M, int N, int K) {
    const int R = M <= 8 ? 8 : 4, groups = ceil_div(M, 16);
    const float rounds = (float)ceil_div(N, R * stream_groups(N, R)) / (2.f * sm_count()), mb = 4e-6f * N * K;
    return 2.f + groups * (rounds * (M <= 4 ? 0.8f : M <= 8 ? 1.f : 1.5f) + mb * (M <= 4 ? 0.18f : M <= 8 ? 0.24f : 0.36f));
}

template <int R, int MM>
static int mm_stream_run(StreamParams p, cudaStream_t st) {
    p.wr = stream_groups(p.N, R);
    launch_dependent(mm_stream_f32_kernel<R, MM>, dim3(ceil_div(p.N, R * p.wr), ceil_div(p.M, MM)), MW_WARPS * 32, 0, st, p);
    return launch_status("bn_linear_f32_stream");
}

}  // namespace bn

using namespace bn;

extern "C" int bn_linear_f32_stream(const float* a, int64_t a_ld, const float* w, int64_t w_ld, const float* bias, int act, float* c,
                                    int64_t c_ld, int M, int N, int K, bn_stream_t stream) {
    const char* what = "bn_linear_f32_stream";
    if (!a || !w || !c) return fail(BN_ERR_INVALID_ARG, "%s: null pointer", what);
    if (M < 0 || N < 0 || N % 8 || K <= 0 || K % 4 || a_ld % 4 || w_ld % 4 || act < 0 || act > BN_ACT_LAST)
        return fail(BN_ERR_INVALID_ARG, "%s: bad shape M=%d N=%d K=%d act=%d", what, M, N, K, act);
    if ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w)) & 15) return fail(BN_ERR_INVALID_ARG, "%s: alignment", what);
    if (M > 65535 * 16) return fail(BN_ERR_UNSUPPORTED, "%s: M=%d too large", what, M);
    if (int rc = require_sm100()) return rc;
    if (M == 0 || N == 0) return BN_OK;
    const StreamParams p{a, w, bias, c, a_ld, w_ld, c_ld, M, N, K, act, 1};
    cudaStream_t st = as_stream(stream);
    if (M <= 2) return mm_stream_run<8, 2>(p, st);
    if (M <= 4) return mm_stream_run<8, 4>(p, st);
    if (M <= 8) return mm_stream_run<8, 8>(p, st);
    return mm_stream_run<4, 16>(p, st);
}
