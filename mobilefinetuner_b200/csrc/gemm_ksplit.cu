// bf16 "NT" tcgen05 GEMM for outputs of few tiles: K is cut over the CTAs of a cluster.
//     D[m,n] = alpha * ( A[m,:K].B[n,:K] + A2[m,:K2].B2[n,:K2] ) + bias[n]          D bf16
//
// A training step of a few hundred to a few thousand tokens has projections of 4 x 9 output tiles under a K of 108 or
// 216 blocks, and LoRA panel products of 4 x 1 tiles: one CTA (pair) per tile leaves most of the 148 SMs idle behind a
// serial K loop.  Here the S = 2 .. 8 CTAs of a cluster take a K range of the same 128 x BN tile each.  When the ranges are
// done the epilogue warps push the f32 partial tiles from tensor memory straight into shared memory of the CTAs that own
// the columns (8-column groups dealt to the ranks; the pipeline stages serve as the exchange area), and every owner adds
// its S slices in rank order and stores bf16.  No workspace, no atomics, one launch, and the result does not depend on timing.
//
// A k-block of a 128 x 128 tile takes 0.30 us, about 570 clocks for its 32 KB: 57 bytes a clock into each SM, where a copy-only
// kernel brings in 72 (microbench tma).  The two cluster barriers and the exchange add about 3 us.  ksplit_plan() weighs that
// against the tile counts of the other kernels.  Measured per launch (20 in a graph, operands rotating over more than the L2):
//     512 x 1152 x 13824   67.3 -> 27.9 us        512 x 768 x 3072   19.8 -> 11.3 us
//     512 x 1152 x  6912   37.2 -> 18.6           512 x 896 x 4864   28.0 -> 13.7
//     512 x   32 x 13824   55.0 -> 12.9          4096 x  16 x 6912   30.2 -> 15.2
#include <cuda.h>

#include <atomic>

#include "common.cuh"
#include "gemm_sm100.h"
#include "sm100_ptx.cuh"

namespace mft {

using namespace ptx;

namespace {

constexpr int BM = 128, BK = 64, EPI_WARPS = 8, THREADS = 64 + 32 * EPI_WARPS, MAX_SPLIT = 8;

template <int BN>
struct KsCfg {
    static constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
    static constexpr int STAGES = BN == 128 ? 6 : 8;
    static constexpr int GROUPS = BN / 8;                         // 8-column groups of a tile, dealt to the ranks
    // the exchange takes over the pipeline's memory: [source rank][group of the slice][half][row] float4; the 129th row
    // shifts neighbouring halves by one bank group, so that a warp can read one row's groups without conflicts
    static constexpr int EX_ROWS = BM + 1;
    static_assert((BN / 8 + MAX_SPLIT) * 2 * EX_ROWS * 16 <= STAGES * STAGE_BYTES, "exchange area");     // S * ceil(GROUPS / S) <= GROUPS + S
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;
};

__device__ __forceinline__ void ks_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_cluster_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

__device__ __forceinline__ void st_cluster_u32(uint32_t addr, uint32_t v) { asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }

// eight columns of one output row
__device__ __forceinline__ void store_cols8(const GemmParams& p, int row, int col, float (&v)[8]) {
    if (row >= p.m || col >= p.n) return;
    __nv_bfloat16* d = static_cast<__nv_bfloat16*>(p.d) + (long long)row * p.ldd + col;
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] *= p.alpha;
    if (p.bias) {
#pragma unroll
        for (int j = 0; j < 8; ++j) if (col + j < p.n) v[j] += __ldg(p.bias + col + j);
    }
    if (col + 8 <= p.n) store8(d, v);
    else
        for (int j = 0; j < 8; ++j) if (col + j < p.n) d[j] = f32_to_bf16(v[j]);
}

template <int BN>
__global__ void __launch_bounds__(THREADS, 1)
gemm_nt_ksplit_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                      const __grid_constant__ CUtensorMap map_a2, const __grid_constant__ CUtensorMap map_b2, const GemmParams p) {
    dep_trigger();
    using Cfg = KsCfg<BN>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(tiles + Cfg::STAGES * Cfg::STAGE_BYTES);
    uint64_t* full_bar = bars;
    uint64_t* empty_bar = bars + Cfg::STAGES;
    uint64_t* tmem_full_bar = bars + 2 * Cfg::STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_full_bar + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* cluster_failed = abort_flag + 1;      // some CTA of the cluster gave up: set by that CTA in all of them

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int splits = p.splits, rank = (int)(blockIdx.x % splits), tile = (int)(blockIdx.x / splits);
    const int m0 = tile_m(tile, p) * BM, n0 = tile_n(tile, p) * BN;
    const int num_kb_main = (p.k + BK - 1) / BK, num_kb = num_kb_main + (p.k2 > 0 ? 1 : 0);
    const int kb0 = (int)((long long)rank * num_kb / splits), kb1 = (int)((long long)(rank + 1) * num_kb / splits);   // never empty: splits <= num_kb

    if (threadIdx.x == 0) {
        for (int s = 0; s < Cfg::STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
        mbar_init(tmem_full_bar, 1);
        *abort_flag = 0;
        *cluster_failed = 0;
        fence_barrier_init();
        tma_prefetch_desc(&map_a); tma_prefetch_desc(&map_b);
        if (p.k2 > 0) { tma_prefetch_desc(&map_a2); tma_prefetch_desc(&map_b2); }
    }
    if (warp == 1) { tmem_alloc(tmem_slot, BN); tmem_relinquish(); }
    tc_fence_before();
    ks_cluster_sync();          // every CTA of the cluster runs before anyone writes into its shared memory
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    dep_wait();                 // set-up above overlapped the previous kernel's tail

    if (warp == 0) {
        if (lane == 0) {
            int stage = 0; uint32_t phase = 0;
            for (int kb = kb0; kb < kb1; ++kb) {
                if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag)) break;
                uint8_t* sa = tiles + stage * Cfg::STAGE_BYTES;
                mbar_arrive_expect_tx(&full_bar[stage], Cfg::STAGE_BYTES);
                const bool main_kb = kb < num_kb_main;
                const int k0 = main_kb ? kb * BK : 0;
                tma_load_2d(sa, main_kb ? &map_a : &map_a2, &full_bar[stage], k0, m0);
                tma_load_2d(sa + Cfg::A_BYTES, main_kb ? &map_b : &map_b2, &full_bar[stage], k0, n0);
                if (++stage == Cfg::STAGES) { stage = 0; phase ^= 1; }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        int stage = 0; uint32_t phase = 0;
        bool ok = true;
        // a ragged last column tile issues narrower MMAs (existing columns rounded up to 16)
        const uint32_t idesc = idesc_bf16_f32(BM, (uint32_t)min(BN, (p.n - n0 + 15) & ~15));
        const uint64_t desc0 = smem_desc_sw128(smem_u32(tiles));
        int kb = kb0;
        for (; kb < kb1; ++kb) {
            if (!__all_sync(0xffffffffu, mbar_wait(&full_bar[stage], phase, abort_flag))) { ok = false; break; }
            tc_fence_after();
            const uint64_t adesc = desc0 + (uint64_t)(stage * (Cfg::STAGE_BYTES >> 4)), bdesc = adesc + (Cfg::A_BYTES >> 4);
            const int nmma = ((kb < num_kb_main ? min(BK, p.k - kb * BK) : p.k2) + 15) / 16;
            if (elect_one()) {
                if (nmma == 4) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) umma_bf16(tmem_base, adesc + 2 * j, bdesc + 2 * j, idesc, (kb > kb0 || j != 0) ? 1u : 0u);
                } else {
                    for (int j = 0; j < nmma; ++j) umma_bf16(tmem_base, adesc + 2 * j, bdesc + 2 * j, idesc, (kb > kb0 || j != 0) ? 1u : 0u);
                }
                umma_commit(&empty_bar[stage]);
            }
            __syncwarp();
            if (++stage == Cfg::STAGES) { stage = 0; phase ^= 1; }
        }
        // the stages become the cluster's exchange area: no load of this CTA may land in them after a wait ran out.  What can
        // be in flight then are the loads from the k-block that did not come on, at most one per stage.
        if (!ok) drain_loads(full_bar, Cfg::STAGES, kb - kb0, min(kb1 - kb0, kb - kb0 + Cfg::STAGES));
        if (ok && elect_one()) umma_commit(tmem_full_bar);
        __syncwarp();
    }
    // ------------------------------------------------ epilogue: warps 2..9, two per lane quarter of tensor memory
    const int q = warp & 3, side = (warp - 2) >> 2, row_in_tile = q * 32 + lane;
    const bool epi = warp >= 2;
    bool landed = false;
    if (epi) {
        landed = __all_sync(0xffffffffu, mbar_wait(tmem_full_bar, 0, abort_flag)) != 0;
        tc_fence_after();
    }
    constexpr int G = Cfg::GROUPS;
    const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16);
    const int groups_n = min(G, (p.n - n0 + 7) / 8);           // groups that exist
    // every MMA of the cluster has read its operands: the stages of all CTAs may be overwritten
    ks_cluster_sync();
    if (threadIdx.x < splits && *abort_flag) st_cluster_u32(map_rank(smem_u32(const_cast<int*>(cluster_failed)), threadIdx.x), 1u);
    const int per_src = ((G + splits - 1) / splits) * 2 * Cfg::EX_ROWS;      // float4 per source rank
    if (epi && landed) {
        const uint32_t ex = smem_u32(tiles) + (uint32_t)((rank * per_src + row_in_tile) * 16);
        int owner = (side * (G / 2) * splits) / G;
        while (owner + 1 < splits && (owner + 1) * G / splits <= side * (G / 2)) ++owner;
#pragma unroll 1
        for (int c = side * (BN / 2); c < (side + 1) * (BN / 2) && n0 + c < p.n; c += 32) {
            uint32_t r[32];
            tmem_ld_32x32(taddr + (uint32_t)c, r);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int g = c / 8 + j;
                if (g >= groups_n) break;
                while (owner + 1 < splits && (owner + 1) * G / splits <= g) ++owner;
                const uint32_t off = (uint32_t)((g - owner * G / splits) * 2 * Cfg::EX_ROWS * 16);
                const uint32_t dst = map_rank(ex + off, (uint32_t)owner);
                // lanes are consecutive rows: 16-byte words side by side, no bank conflicts
                st_cluster_v4(dst, r[8 * j], r[8 * j + 1], r[8 * j + 2], r[8 * j + 3]);
                st_cluster_v4(dst + Cfg::EX_ROWS * 16, r[8 * j + 4], r[8 * j + 5], r[8 * j + 6], r[8 * j + 7]);
            }
        }
    }
    __syncwarp();
    ks_cluster_sync();
    if (*cluster_failed == 0) {                 // (a rank that gave up sent nothing: the exchange area holds operand bytes in its place)
        const int g0 = rank * G / splits, ng = min((rank + 1) * G / splits, groups_n) - g0;
        const float4* ex = reinterpret_cast<const float4*>(tiles);
        // consecutive threads: consecutive groups of a row (contiguous bytes of D)
        for (int i = threadIdx.x; ng > 0 && i < BM * ng; i += THREADS) {
            const int row = i / ng, g = i - row * ng;
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = 0.f;
            for (int s = 0; s < splits; ++s) {
                const float4* src = ex + s * per_src + g * 2 * Cfg::EX_ROWS + row;
                const float4 a = src[0], b = src[Cfg::EX_ROWS];
                v[0] += a.x; v[1] += a.y; v[2] += a.z; v[3] += a.w;
                v[4] += b.x; v[5] += b.y; v[6] += b.z; v[7] += b.w;
            }
            store_cols8(p, m0 + row, n0 + (g0 + g) * 8, v);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag && p.status) atomicExch(p.status, MFT_ERR_TIMEOUT);
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, BN);
    }
}

template <int BN>
int32_t launch(const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& ma2, const CUtensorMap& mb2, GemmParams p, cudaStream_t stream) {
    using Cfg = KsCfg<BN>;
    static PerDeviceFlag configured_on;
    bool& configured = configured_on.here();
    if (!configured) {
        if (int32_t s = check_cuda(cudaFuncSetAttribute(gemm_nt_ksplit_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES), "gemm ksplit smem attr")) return s;
        configured = true;
    }
    p.num_m_tiles = (p.m + BM - 1) / BM;
    p.num_n_tiles = (p.n + BN - 1) / BN;
    p.tiles_mn = p.num_m_tiles * p.num_n_tiles;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(p.tiles_mn * p.splits));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = Cfg::SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)p.splits; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = dep_launch_enabled() ? 2 : 1;
    cudaLaunchKernelEx(&cfg, gemm_nt_ksplit_kernel<BN>, ma, mb, ma2, mb2, p);
    MFT_LAUNCH_CHECK("gemm_nt");
    return MFT_OK;
}

}  // namespace

// Clusters of S CTAs that run at the same time on this device: the SMs of a GPC come in pairs that S has to fit into, so the
// count is the driver's answer (B200: 74 of 2, 33 of 4, 15 of 8), asked once per device.  0: the driver gives none or no answer,
// and no plan has clusters of this size.  Threads that ask at the same time write the same value.
static int active_clusters(int dev, int bn, int s) {
    constexpr int NOT_ASKED = 0, NONE = -1, DEVICES = 64;
    static std::atomic<int> known[DEVICES][2][MAX_SPLIT + 1] = {};
    if (dev < 0 || dev >= DEVICES) return 0;
    std::atomic<int>& entry = known[dev][bn == 128][s];
    const int seen = entry.load(std::memory_order_relaxed);
    if (seen != NOT_ASKED) return seen == NONE ? 0 : seen;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(num_sms() / s * s));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = bn == 128 ? KsCfg<128>::SMEM_BYTES : KsCfg<64>::SMEM_BYTES;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)s; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int got = 0;
    cudaError_t e = bn == 128 ? cudaFuncSetAttribute(gemm_nt_ksplit_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, KsCfg<128>::SMEM_BYTES)
                              : cudaFuncSetAttribute(gemm_nt_ksplit_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, KsCfg<64>::SMEM_BYTES);
    if (e == cudaSuccess)
        e = bn == 128 ? cudaOccupancyMaxActiveClusters(&got, gemm_nt_ksplit_kernel<128>, &cfg) : cudaOccupancyMaxActiveClusters(&got, gemm_nt_ksplit_kernel<64>, &cfg);
    if (e != cudaSuccess) { got = 0; cudaGetLastError(); }
    entry.store(got > 0 ? got : NONE, std::memory_order_relaxed);
    return got > 0 ? got : 0;
}

// Tile width (64 or 128; 0 = not this kernel) and K ranges for a bf16 plain-store call of this shape.  Times in ns.
KsplitPlan ksplit_plan(int64_t m, int64_t n, int64_t k, int64_t k2) {
    KsplitPlan best;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) { cudaGetLastError(); return best; }
    const int64_t sms = num_sms(), kb = (k + BK - 1) / BK + (k2 > 0 ? 1 : 0);
    // what the persistent kernels take (measured on launches of one wave): 300 ns per k-block of a 256 x 256 pair tile,
    // 270 ns of a 128 x 64 single-CTA tile, plus the end of the last tile
    double other;
    if (m >= 256 && n >= 192) {
        const int64_t tiles = ((m + 255) / 256) * ((n + 255) / 256), waves = (tiles + sms / 2 - 1) / (sms / 2);
        other = (double)waves * ((double)kb * 300.0 + 1000.0) + 5200.0;
    } else {
        const int64_t tiles = ((m + BM - 1) / BM) * ((n + 63) / 64), waves = (tiles + sms - 1) / sms;
        other = (double)waves * ((double)kb * 270.0 + 500.0) + 2600.0;
    }
    double best_cost = 0.95 * other;
    for (int bn = 128; bn >= 64; bn -= 64) {
        if (bn == 128 && n <= 64) continue;
        const int64_t tiles = ((m + BM - 1) / BM) * ((n + bn - 1) / bn);
        for (int sp = 2; sp <= MAX_SPLIT && kb / sp >= 4; ++sp) {      // (shorter ranges gain less than the exchange costs)
            const int64_t clusters = active_clusters(dev, bn, sp);
            if (tiles > clusters) continue;             // one tile per CTA: a second wave repeats the start-up
            const double cost = (double)((kb + sp - 1) / sp) * (bn == 128 ? 300.0 : 270.0) + (bn == 128 ? 6500.0 : 5000.0);
            if (cost < best_cost) { best_cost = cost; best = {bn, sp}; }
        }
    }
    return best;
}

int32_t gemm_nt_run_ksplit(const GemmCall& c, cudaStream_t stream) {
    const bool ok = c.epi == EPI_STORE && !c.d_is_f32 && !c.accumulate && c.splits <= 1 && c.a && c.b && c.d && c.m > 0 && c.n > 0 && c.k > 0 &&
                    c.m < (1 << 30) && c.n < (1 << 30) && c.k < (1 << 30) && c.k2 >= 0 && c.k2 <= BK && (c.k2 == 0 || (c.a2 && c.b2)) &&
                    c.ldd >= c.n && c.lda >= c.k && c.ldb >= c.k && c.ldd % 8 == 0 && reinterpret_cast<uintptr_t>(c.d) % 16 == 0;
    if (!ok) return MFT_ERR_UNSUPPORTED;
    const KsplitPlan plan = ksplit_plan(c.m, c.n, c.k, c.k2);
    if (plan.bn == 0) return MFT_ERR_UNSUPPORTED;
    CUtensorMap ma, mb, ma2, mb2;
    if (int32_t s = make_tmap_bf16(&ma, c.a, c.m, c.k, c.lda, BM)) return s;
    if (int32_t s = make_tmap_bf16(&mb, c.b, c.n, c.k, c.ldb, plan.bn)) return s;
    ma2 = ma; mb2 = mb;
    if (c.k2 > 0) {
        if (int32_t s = make_tmap_bf16(&ma2, c.a2, c.m, c.k2, c.lda2, BM)) return s;
        if (int32_t s = make_tmap_bf16(&mb2, c.b2, c.n, c.k2, c.ldb2, plan.bn)) return s;
    }
    GemmParams p{};
    p.m = (int)c.m; p.n = (int)c.n; p.k = (int)c.k; p.k2 = (int)c.k2;
    p.alpha = c.alpha; p.bias = c.bias; p.d = c.d; p.ldd = c.ldd;
    p.splits = plan.splits;
    p.status = device_status_word();
    return plan.bn == 128 ? launch<128>(ma, mb, ma2, mb2, p, stream) : launch<64>(ma, mb, ma2, mb2, p, stream);
}

}  // namespace mft
