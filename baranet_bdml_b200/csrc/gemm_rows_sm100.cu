// C (M,N) bf16 = A (M,K) @ W (N,K)^T for 17 to 128 rows: a step of that many sequences, one token each.
//
// What such a product costs is the weights' way through the chip, so all multiprocessors have to take part in it from the
// start, and nothing else should pass through memory.  The weights are the MMA's 128-row operand and the rows of A its narrow
// one (N = 32, 64 or 128): a stage of 64 k holds 16 KB of weights beside 4 - 16 KB of A.  A cluster of up to eight CTAs shares
// an output tile, each with a range of K, and adds up through distributed shared memory in rank order; no partial sum goes to
// global memory and there is no second launch.  Two CTAs fit on a multiprocessor (of gate and up of more than 64 rows one), so that
// most shapes are one wave.
// A programmatic dependent: while the kernel ahead finishes, every CTA asks for all of its weights in L2.
//
// Epilogues: bf16, the fp32 sum, act(sum + bias), act(sum) * factor, act(gate) * up (two weight tiles, two accumulators).
// Warps 0-3 read the accumulator (lane = output column), all six add up and store; warp 4 issues MMAs, warp 5 loads by TMA.
#include "gemm_rows.cuh"
#include "hybrid.cuh"
#include "ptx.cuh"
#include "tcgen05.cuh"
#include "tma.cuh"

namespace bn {

using namespace ptx;

constexpr int GR_BN = 128, GR_BK = 64, GR_THREADS = 192, GR_MAX_CLUSTER = 8;

// MT: rows that the tile has room for.  NW: weight tiles (2: gate and up)
template <int MT, int NW> struct RowsShape {
    static constexpr int W_BYTES = GR_BN * GR_BK * 2, A_BYTES = MT * GR_BK * 2, STAGE_BYTES = NW * W_BYTES + A_BYTES;
    static constexpr int NSTAGE = 106496 / STAGE_BYTES;
    static constexpr int LDP = GR_BN + 4;                                  // row stride of the sums, floats
    static constexpr int RING = NSTAGE * STAGE_BYTES, SUMS = NW * MT * LDP * 4;
    static constexpr int SMEM_BYTES = 1024 + (RING > SUMS ? RING : SUMS);
    static constexpr int PER_SM = SMEM_BYTES <= 113 * 1024 ? 2 : 1;        // of 228 KB, 1 of them the system's for each CTA
    static constexpr uint32_t TMEM_COLS = NW * MT < 32 ? 32 : NW * MT;
};

__device__ __forceinline__ float4 ld_cluster(uint32_t addr, uint32_t rank) {
    float4 v;
    asm volatile(
        "{\n\t.reg .b32 r;\n\t"
        "mapa.shared::cluster.u32 r, %4, %5;\n\t"
        "ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [r];\n\t}"
        : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
        : "r"(addr), "r"(rank)
        : "memory");
    return v;
}

template <int MT, int NW>
__global__ void __launch_bounds__(GR_THREADS)
gemm_rows_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_a, const RowsGemm p, int ranks,
                 int k_per_rank) {
    using Sh = RowsShape<MT, NW>;
    constexpr int NSTAGE = Sh::NSTAGE;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bar_full[NSTAGE], bar_empty[NSTAGE], bar_done;
    __shared__ uint32_t s_tmem_base;
    __shared__ int s_abort;

    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int rank = blockIdx.x % ranks, n0 = blockIdx.x / ranks * GR_BN;     // n0: first output column
    const int k_steps = (p.K + GR_BK - 1) / GR_BK, ks0 = min(rank * k_per_rank, k_steps), ks1 = min(k_steps, ks0 + k_per_rank);

    if (tid == 0) {
        for (int s = 0; s < NSTAGE; ++s) {
            mbar_init(smem_u32(&bar_full[s]), 1);
            mbar_init(smem_u32(&bar_empty[s]), 1);
        }
        mbar_init(smem_u32(&bar_done), 1);
        s_abort = 0;
        fence_mbar_init();
    }
    if (warp == 4) {
        tc::tmem_alloc(smem_u32(&s_tmem_base), Sh::TMEM_COLS);
        tc::tmem_relinquish();
    }
    if (warp == 5 && lane == 0) {
        prefetch_tensormap(&tmap_w);
        prefetch_tensormap(&tmap_a);
        for (int ks = ks0; ks < ks1; ++ks)
#pragma unroll
            for (int q = 0; q < NW; ++q) tma_prefetch_2d(&tmap_w, ks * GR_BK, NW * n0 + q * GR_BN);
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = s_tmem_base;
    grid_launch_dependents();
    grid_dependency_wait();

    if (warp == 5) {
        if (lane == 0) {
            bool ok = true;
            for (int ks = ks0; ok && ks < ks1; ++ks) {
                const int it = ks - ks0, stage = it % NSTAGE;
                ok = mbar_wait(smem_u32(&bar_empty[stage]), ((it / NSTAGE) & 1u) ^ 1u, &s_abort);
                if (!ok) break;
                const uint32_t full = smem_u32(&bar_full[stage]), sW = smem0 + stage * Sh::STAGE_BYTES;
                mbar_arrive_expect_tx(full, Sh::STAGE_BYTES);
#pragma unroll
                for (int q = 0; q < NW; ++q) tma_load_2d(sW + q * Sh::W_BYTES, &tmap_w, ks * GR_BK, NW * n0 + q * GR_BN, full);
                tma_load_2d(sW + NW * Sh::W_BYTES, &tmap_a, ks * GR_BK, 0, full);
            }
        }
        __syncwarp();
    } else if (warp == 4) {
        constexpr uint32_t IDESC = tc::idesc_bf16(GR_BN, MT, 0);
        const uint64_t d0 = tc::smem_desc_sw128(0);
        bool ok = true;
        for (int ks = ks0; ks < ks1; ++ks) {
            const int it = ks - ks0, stage = it % NSTAGE;
            ok = mbar_wait(smem_u32(&bar_full[stage]), (it / NSTAGE) & 1u, &s_abort);
            if (!ok) break;
            if (elect_one()) {
                tc::fence_after_sync();
                const uint32_t sW = smem0 + stage * Sh::STAGE_BYTES, sA = sW + NW * Sh::W_BYTES;
#pragma unroll
                for (int q = 0; q < NW; ++q)
#pragma unroll
                    for (int kk = 0; kk < GR_BK / 16; ++kk)
                        tc::mma_ss(tmem + q * MT, d0 + (uint64_t)(((sW + q * Sh::W_BYTES) >> 4) + kk * 2), d0 + (uint64_t)((sA >> 4) + kk * 2),
                                   IDESC, it > 0 || kk > 0);
                tc::commit(smem_u32(&bar_empty[stage]));
                if (ks == ks1 - 1) tc::commit(smem_u32(&bar_done));
            }
            __syncwarp();
        }
    }
    // All MMAs of this CTA have read their stages when bar_done completes: its sums take the ring's place, [row][column]
    float* sums = reinterpret_cast<float*>(smem_raw + (smem0 - smem_u32(smem_raw)));
    if (warp < 4) {
        const bool some = ks1 > ks0;
        const bool ok = !some || mbar_wait(smem_u32(&bar_done), 0, &s_abort);
        __syncwarp();
        if (ok) {
            tc::fence_after_sync();
#pragma unroll
            for (int q = 0; q < NW; ++q)
#pragma unroll
                for (int c = 0; c < MT / 32; ++c) {
                    uint32_t r[32];
                    if (some) {
                        tc::ld32(tmem + ((uint32_t)(warp * 32) << 16) + q * MT + c * 32, r);
                        tc::wait_ld(r);
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i) r[i] = 0;
                    }
#pragma unroll
                    for (int i = 0; i < 32; ++i) sums[(q * MT + c * 32 + i) * Sh::LDP + tid] = __uint_as_float(r[i]);
                }
        }
        tc::fence_before_sync();
    }
    cluster_sync();
    // a rank finishes the rows rank, rank + ranks, ...; a warp has a whole row of the tile, four columns a lane
    const int n = n0 + lane * 4;
    const uint32_t mine = smem0 + lane * 16;
    if (n < p.n_out)                                           // a multiple of 8
        for (int m = rank + warp * ranks; m < p.M; m += ranks * (GR_THREADS / 32)) {
            // all ranks' loads ahead of the first addition: each is a trip to another multiprocessor
            float4 part[GR_MAX_CLUSTER][NW];
#pragma unroll
            for (int r = 0; r < GR_MAX_CLUSTER; ++r)
                if (r < ranks)
#pragma unroll
                    for (int q = 0; q < NW; ++q) part[r][q] = ld_cluster(mine + (q * MT + m) * Sh::LDP * 4, r);
            float v[NW][4];
#pragma unroll
            for (int q = 0; q < NW; ++q) v[q][0] = v[q][1] = v[q][2] = v[q][3] = 0.f;
#pragma unroll
            for (int r = 0; r < GR_MAX_CLUSTER; ++r)
                if (r < ranks)
#pragma unroll
                    for (int q = 0; q < NW; ++q) {
                        v[q][0] += part[r][q].x; v[q][1] += part[r][q].y; v[q][2] += part[r][q].z; v[q][3] += part[r][q].w;
                    }
            if (p.c32) {
                store4(p.c32 + (size_t)m * p.n_out + n, v[0]);
                continue;
            }
            float f[4] = {1.f, 1.f, 1.f, 1.f};
            if (p.bias) load4(p.bias + n, f);
            if (p.mul) load4(p.mul + (size_t)m * p.mul_ld + n, f);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (NW == 2) v[0][e] = activation_fast(p.act, v[0][e]) * v[NW - 1][e];
                else if (p.mul) v[0][e] = activation_fast(p.act, v[0][e]) * f[e];
                else v[0][e] = activation_fast(p.act, p.bias ? v[0][e] + f[e] : v[0][e]);
            }
            store4(p.c + (size_t)m * p.n_out + n, v[0]);
        }
    cluster_sync();                                            // nobody leaves while its sums are being read
    __syncwarp();
    if (tid == 0 && s_abort && p.error_word) atomicExch(p.error_word, BN_ERR_TIMEOUT);
    if (warp == 4) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem, Sh::TMEM_COLS);
    }
}

// How many CTAs run together: one or two per multiprocessor, as their shared memory fits (gate and up of more than 64 rows: one),
// less what whole clusters do not fill (measured with two: 252 to 268 CTAs run together, 288 do not).
static int rows_resident(int per_sm) { return per_sm == 2 ? sm_count() * 9 / 5 + 2 : sm_count() * 9 / 10; }

// CTAs per output tile: the most, an even number, of which the GPU runs all at the same time and that have 5 steps of 64 k each
// (gemm_rows_ok: two of them always are).
// 64 rows, us by ranks (2, 4, 6, 8): 2048 -> 4608 11.0, 9.1, 8.5, 12.8; 2048 -> 7424 13.0, 9.9, 14.4, 15.8; 2048 -> 2048 8.8, 6.2,
// 5.9, 6.8; 7424 -> 2048 19.6, 13.6, 12.3, 12.1.
// 64-wide tiles of 128 rows of A, K over single CTAs and a second launch for the sums took 12.7, 15.1, 9.7, 17.3 us (a weight of
// 30 MB alone 4.7 us).
static int rows_ranks(int tiles, int steps, int resident) {
    int r = GR_MAX_CLUSTER;
    while (r > 2 && (tiles * r > resident || steps < 5 * r)) r -= 2;
    return r;
}

// - With more tiles than half of what runs together 128 x 256 tiles do as well: 2048 -> 32000, 64 rows, 28.7 us there, 30.6 here.
// - A short K leaves a tile to one or two CTAs, and the time is that of the sums' way, which grows with the rows: 256 -> 2048, 17 /
//   64 / 128 rows, 4.2 / 6.7 / 10.2 us here, 4.5 / 4.7 / 5.9 as 128 x 256 tiles; 512 -> 8192 5.7 / 8.2 / 11.9, there 5.9 / 6.1 /
//   7.2; 640 -> 2048 4.3 / 6.1 / 8.0, there 6.3 / 6.4 / 7.6, and with K over single CTAs 6.2 / 6.5 / 7.1; 1024 -> 2048 4.9 / 6.8 /
//   8.8, that form 7.1 / 6.9 / 7.5; 2048 -> 2048 128 rows 8.8, that form 9.7.
// - Gate and up take twice the shared memory and twice that way, and are faster than 256-wide tiles of both where four CTAs share a
//   tile, or two and the rows are few: 2048 -> 5632, four CTAs, 17 / 64 rows 12.0 / 15.0 us, there 18.1, and two CTAs, 65 / 128 rows,
//   18.4 / 20.7; 2048 -> 2816 65 / 128 rows 10.8 / 12.8, there 17.1; 2048 -> 8704, two CTAs, 17 / 64 rows 22.1 / 24.2, there 20.1;
//   1024 -> 4096, two CTAs, 17 / 48 / 64 / 128 rows 9.6 / 11.2 / 12.1 / 13.7, there 11.4.
bool gemm_rows_ok(int M, int n_out, int K, bool glu) {
    if (M > GR_MAX_ROWS || K < 640) return false;
    const int tiles = ceil_div(n_out, GR_BN);
    if (!glu) return tiles * 2 <= rows_resident(2) && (M <= 64 || K >= 1280);
    return tiles * 4 <= rows_resident(M <= 64 ? 2 : 1) && (M <= 48 || K >= 1280);
}

template <int MT, int NW>
static int rows_launch(const RowsGemm& p, cudaStream_t st, const char* what) {
    using Sh = RowsShape<MT, NW>;
    static thread_local int configured_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (configured_dev != dev) {
        cudaError_t e = cudaFuncSetAttribute(gemm_rows_kernel<MT, NW>, cudaFuncAttributeMaxDynamicSharedMemorySize, Sh::SMEM_BYTES);
        if (e != cudaSuccess) return fail(BN_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
        configured_dev = dev;
    }
    CUtensorMap mw, ma;
    const uint64_t dims_w[2] = {(uint64_t)p.K, (uint64_t)p.N}, dims_a[2] = {(uint64_t)p.K, (uint64_t)p.M}, stride[1] = {(uint64_t)p.K * 2};
    const uint32_t box_w[2] = {GR_BK, GR_BN}, box_a[2] = {GR_BK, MT};
    if (int rc = make_tensor_map(&mw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, p.w, dims_w, stride, box_w, CU_TENSOR_MAP_SWIZZLE_128B)) return rc;
    if (int rc = make_tensor_map(&ma, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, p.a, dims_a, stride, box_a, CU_TENSOR_MAP_SWIZZLE_128B)) return rc;
    const int tiles = (p.n_out + GR_BN - 1) / GR_BN, steps = (p.K + GR_BK - 1) / GR_BK;
    const int ranks = rows_ranks(tiles, steps, rows_resident(Sh::PER_SM));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles * ranks));
    cfg.blockDim = dim3(GR_THREADS);
    cfg.dynamicSmemBytes = Sh::SMEM_BYTES;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)ranks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    cudaError_t e = launch_config(cfg, 1, gemm_rows_kernel<MT, NW>, mw, ma, p, ranks, (steps + ranks - 1) / ranks);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return fail(BN_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
    }
    return launch_status(what);
}

int gemm_rows(const RowsGemm& p, cudaStream_t st, const char* what) {
    if (p.glu) return p.M <= 32 ? rows_launch<32, 2>(p, st, what) : p.M <= 64 ? rows_launch<64, 2>(p, st, what) : rows_launch<128, 2>(p, st, what);
    return p.M <= 32 ? rows_launch<32, 1>(p, st, what) : p.M <= 64 ? rows_launch<64, 1>(p, st, what) : rows_launch<128, 1>(p, st, what);
}

}  // namespace bn
