// Batched f32 matrix product behind the eager operators: C[b] = A[b] (M x K) * op(B[b]), B stored [K,N] or [N,K].
// The operators promise f32 accuracy, so the products run on the CUDA cores in f32 FMAs.
//
// What bounds it: the FMA pipes (128 lanes per SM, 74 TFLOP/s over the chip at 1.965 GHz).  Each thread keeps an 8 x 8 block of C in
// registers, so one k step is 64 FMAs against four 16-byte shared-memory reads (a warp covers 32 x 64 of the tile in a
// 4 x 8 thread grid: 4 and 8 distinct 16-byte words per read, one shared-memory wavefront each).  The next k slab is on
// its way from global memory to registers while the current one is multiplied.
//
// Tiles: 128 x 128 (8 warps) where that fills the chip, 64 x 64 (2 warps) otherwise; a short output under a long K is
// also cut along K over the CTAs of a cluster (up to 8), which add their partial tiles through distributed shared
// memory in rank order, so the result does not depend on timing.  plan() below picks by the FMA time of the SM that gets
// the most work.
//
// A product of at most one or two 32 x 32 tiles per SM under a short K goes to matmul_f32_small_kernel: see small_tiles().
//
// Measured: 4096^3 48.8 TFLOP/s, 512 x 4864 x 896 28.6 and 512 x 896 x 4864 27.5; one output per thread on 32 x 32 tiles
// ran all of them at 5.2 (the f32 gated MLP of 512 tokens at 896 / 4864, forward and backward: 5.13 -> 0.96 ms).
#include <cooperative_groups.h>

#include "common.cuh"
#include "gemm_sm100.h"

namespace mft {
namespace {

namespace cg = cooperative_groups;

constexpr int BK = 16, PAD = 4;
static_assert(BK == 16, "the slab loads deal four float4 of a row to four threads");

template <int BM, int BN>
struct MmCfg {
    static constexpr int THREADS = (BM / 8) * (BN / 8);
    static constexpr int A_LD = BM + PAD, B_LD = BN + PAD;
    static constexpr int STAGE_FLOATS = BK * (A_LD + B_LD);
    static constexpr int A_VEC = BM * BK / 4 / THREADS, B_VEC = BN * BK / 4 / THREADS;    // float4 loads per thread and slab
    static constexpr int SMEM_FLOATS = 2 * STAGE_FLOATS > BM * BN ? 2 * STAGE_FLOATS : BM * BN;
};

// four consecutive floats of a row, zero past `limit` (VEC: the row start and the extent are multiples of four floats)
template <bool VEC>
__device__ __forceinline__ float4 load4(const float* __restrict__ row, int col, int limit, bool row_ok) {
    float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!row_ok) return r;
    if (VEC) {
        if (col < limit) r = __ldg(reinterpret_cast<const float4*>(row + col));
    } else {
        if (col < limit) r.x = __ldg(row + col);
        if (col + 1 < limit) r.y = __ldg(row + col + 1);
        if (col + 2 < limit) r.z = __ldg(row + col + 2);
        if (col + 3 < limit) r.w = __ldg(row + col + 3);
    }
    return r;
}

template <int BM, int BN, bool TRANS_B, bool VEC>
__global__ void __launch_bounds__(MmCfg<BM, BN>::THREADS)
matmul_f32_kernel(const float* __restrict__ A, const float* __restrict__ B, float* __restrict__ C, int M, int N, int K, int n_tiles, int k_per_split,
                  int64_t stride_a, int64_t stride_b, int64_t stride_c) {
    using Cfg = MmCfg<BM, BN>;
    extern __shared__ __align__(16) float smem[];
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    // thread grid: warps are 4 (rows) x 8 (columns) threads; a thread's 8 x 8 block is four 4 x 4 corners of the tile
    constexpr int WCOLS = BN / 64;
    const int ty = (warp / WCOLS) * 4 + (lane >> 3), tx = (warp % WCOLS) * 8 + (lane & 7);
    const int m0 = (int)(blockIdx.x / n_tiles) * BM, n0 = (int)(blockIdx.x % n_tiles) * BN;
    const int kb = blockIdx.y * k_per_split, ke = min(K, kb + k_per_split);
    const float* a = A + blockIdx.z * stride_a;
    const float* b = B + blockIdx.z * stride_b;
    float* c = C + blockIdx.z * stride_c;

    float4 ra[Cfg::A_VEC], rb[Cfg::B_VEC];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < Cfg::A_VEC; ++i) {
            const int v = t + i * Cfg::THREADS, r = m0 + v / 4;
            ra[i] = load4<VEC>(a + (int64_t)r * K, k0 + (v % 4) * 4, ke, r < M);
        }
#pragma unroll
        for (int i = 0; i < Cfg::B_VEC; ++i) {
            const int v = t + i * Cfg::THREADS;
            if (TRANS_B) {
                const int r = n0 + v / 4;
                rb[i] = load4<VEC>(b + (int64_t)r * K, k0 + (v % 4) * 4, ke, r < N);
            } else {
                const int r = k0 + v / (BN / 4);
                rb[i] = load4<VEC>(b + (int64_t)r * N, n0 + (v % (BN / 4)) * 4, N, r < ke);
            }
        }
    };
    auto put = [&](float* stage) {
        float* as = stage;                           // [BK][A_LD], k-major
        float* bs = stage + BK * Cfg::A_LD;          // [BK][B_LD]
#pragma unroll
        for (int i = 0; i < Cfg::A_VEC; ++i) {
            const int v = t + i * Cfg::THREADS, r = v / 4, kk = (v % 4) * 4;
            as[(kk + 0) * Cfg::A_LD + r] = ra[i].x; as[(kk + 1) * Cfg::A_LD + r] = ra[i].y;
            as[(kk + 2) * Cfg::A_LD + r] = ra[i].z; as[(kk + 3) * Cfg::A_LD + r] = ra[i].w;
        }
#pragma unroll
        for (int i = 0; i < Cfg::B_VEC; ++i) {
            const int v = t + i * Cfg::THREADS;
            if (TRANS_B) {
                const int r = v / 4, kk = (v % 4) * 4;
                bs[(kk + 0) * Cfg::B_LD + r] = rb[i].x; bs[(kk + 1) * Cfg::B_LD + r] = rb[i].y;
                bs[(kk + 2) * Cfg::B_LD + r] = rb[i].z; bs[(kk + 3) * Cfg::B_LD + r] = rb[i].w;
            } else {
                *reinterpret_cast<float4*>(bs + (v / (BN / 4)) * Cfg::B_LD + (v % (BN / 4)) * 4) = rb[i];
            }
        }
    };

    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;

    if (kb < ke) { fetch(kb); put(smem); }
    __syncthreads();
    int cur = 0;
    for (int k0 = kb; k0 < ke; k0 += BK) {
        const bool more = k0 + BK < ke;
        if (more) fetch(k0 + BK);
        const float* as = smem + cur * Cfg::STAGE_FLOATS + ty * 4;
        const float* bs = smem + cur * Cfg::STAGE_FLOATS + BK * Cfg::A_LD + tx * 4;
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            float av[8], bv[8];
            *reinterpret_cast<float4*>(av) = *reinterpret_cast<const float4*>(as + k * Cfg::A_LD);
            *reinterpret_cast<float4*>(av + 4) = *reinterpret_cast<const float4*>(as + k * Cfg::A_LD + BM / 2);
            *reinterpret_cast<float4*>(bv) = *reinterpret_cast<const float4*>(bs + k * Cfg::B_LD);
            *reinterpret_cast<float4*>(bv + 4) = *reinterpret_cast<const float4*>(bs + k * Cfg::B_LD + BN / 2);
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
        }
        if (more) put(smem + (cur ^ 1) * Cfg::STAGE_FLOATS);     // the other slab was last read before the previous barrier
        __syncthreads();
        cur ^= 1;
    }

    auto store_row = [&](int row, int col, float4 v) {
        if (row >= M || col >= N) return;
        float* p = c + (int64_t)row * N + col;
        if (VEC) { *reinterpret_cast<float4*>(p) = v; return; }
        p[0] = v.x;
        if (col + 1 < N) p[1] = v.y;
        if (col + 2 < N) p[2] = v.z;
        if (col + 3 < N) p[3] = v.w;
    };
    if (gridDim.y == 1) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int row = m0 + (i & 4 ? BM / 2 : 0) + ty * 4 + (i & 3);
            store_row(row, n0 + tx * 4, make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]));
            store_row(row, n0 + BN / 2 + tx * 4, make_float4(acc[i][4], acc[i][5], acc[i][6], acc[i][7]));
        }
        return;
    }
    // K was cut over the cluster: park the partial tile in shared memory (the slabs are done with), then every rank adds
    // its share of the rows over all ranks
    cg::cluster_group cluster = cg::this_cluster();
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int row = (i & 4 ? BM / 2 : 0) + ty * 4 + (i & 3);
        *reinterpret_cast<float4*>(smem + row * BN + tx * 4) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        *reinterpret_cast<float4*>(smem + row * BN + BN / 2 + tx * 4) = make_float4(acc[i][4], acc[i][5], acc[i][6], acc[i][7]);
    }
    cluster.sync();
    const int ranks = (int)gridDim.y, rank = (int)cluster.block_rank(), rows = BM / ranks;
    for (int v = t; v < rows * BN / 4; v += Cfg::THREADS) {
        const int row = rank * rows + v / (BN / 4), col = (v % (BN / 4)) * 4;
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int r = 0; r < ranks; ++r) {
            const float4 x = *reinterpret_cast<const float4*>(cluster.map_shared_rank(smem, r) + row * BN + col);
            s.x += x.x; s.y += x.y; s.z += x.z; s.w += x.w;
        }
        store_row(m0 + row, n0 + col, s);
    }
    cluster.sync();       // nobody leaves while its partial tile is still being read
}

// One output per thread from 32 x 32 tiles: a small product is bound by the latency of its serial k loop, which 32 warps of
// one FMA and two shared-memory reads a step walk faster than the two warps of a 64 x 64 tile.
__global__ void __launch_bounds__(1024)
matmul_f32_small_kernel(const float* __restrict__ A, const float* __restrict__ B, float* __restrict__ C, int M, int N, int K, int64_t stride_a,
                        int64_t stride_b, int64_t stride_c, int trans_b) {
    __shared__ float as[32][33], bs[32][33];
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int row = blockIdx.y * 32 + ty, n0 = blockIdx.x * 32, col = n0 + tx;
    const float* a = A + blockIdx.z * stride_a;
    const float* b = B + blockIdx.z * stride_b;
    float acc = 0.f;
    for (int k0 = 0; k0 < K; k0 += 32) {
        as[ty][tx] = (row < M && k0 + tx < K) ? a[(int64_t)row * K + k0 + tx] : 0.f;
        if (trans_b) bs[tx][ty] = (k0 + tx < K && n0 + ty < N) ? b[(int64_t)(n0 + ty) * K + k0 + tx] : 0.f;      // rows of B side by side
        else bs[ty][tx] = (k0 + ty < K && col < N) ? b[(int64_t)(k0 + ty) * N + col] : 0.f;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 32; ++k) acc = fmaf(as[ty][k], bs[k][tx], acc);
        __syncthreads();
    }
    if (row < M && col < N) C[blockIdx.z * stride_c + (int64_t)row * N + col] = acc;
}

struct MmPlan { bool big; int splits; };
// FMA time of the busiest SM in units of one 64 x 64 x 1 slab, tiles dealt round to the SMs.  A 64 x 64 tile re-reads
// its operands more often and has two warps to hide latency with: charged 15 %; each extra K range 64 steps for its pass
// through shared memory.
MmPlan plan(int64_t m, int64_t n, int64_t k, int64_t batch) {
    const int64_t sms = num_sms();
    const int64_t big_tiles = ((m + 127) / 128) * ((n + 127) / 128) * batch, small_tiles = ((m + 63) / 64) * ((n + 63) / 64) * batch;
    MmPlan best{true, 1};
    double cost = (double)((big_tiles + sms - 1) / sms) * 4.0 * (double)k;
    for (int sp = 1; sp <= 8; sp *= 2) {
        if (sp > 1 && k / sp < 128) break;
        const double c = (double)((small_tiles * sp + sms - 1) / sms) * 1.15 * (double)((k + sp - 1) / sp + (sp > 1 ? 64 : 0));
        if (c < cost) { cost = c; best = {false, sp}; }
    }
    return best;
}

// Where the 32 x 32 tiles are the faster ones.  Microseconds 32 x 32 / register-blocked for one 128 x 128 product (16 tiles):
//   B [K,N]:  K = 32 3.5 / 5.3,  128 8.1 / 13.3,  256 15 / 16.5,  384 21.6 / 22,  512 28 / 15.6 (cut over a cluster from there on)
//   B [N,K]:  K = 32 3.8 / 5.1,  128 8.3 / 12.5,  192 12 / 17.4,  256 15 / 15.1
// up to one tile per SM.  With two (256 products of 16 x 16), B [K,N] is even or ahead while K is not cut: K = 8 4.9 / 3.6,
// 32 5.0 / 5.1,  64 8.2 / 8.4,  192 19.2 / 20.2,  1024 90.6 / 95.5;  B [N,K] behind: 8.7 / 7.7 at 64.
bool small_tiles(int64_t m, int64_t n, int64_t k, int64_t batch, bool trans_b, const MmPlan& p) {
    const int64_t tiles = ((m + 31) / 32) * ((n + 31) / 32) * batch, sms = num_sms();
    if (tiles <= sms && k < (trans_b ? 256 : 448)) return true;
    return !trans_b && tiles <= 2 * sms && !p.big && p.splits == 1 && k >= 32;
}

template <int BM, int BN, bool TRANS_B, bool VEC>
int32_t launch(const float* a, const float* b, float* c, int64_t batch, int64_t m, int64_t n, int64_t k, int64_t sa, int64_t sb, int64_t sc, int splits,
               cudaStream_t stream) {
    using Cfg = MmCfg<BM, BN>;
    static PerDeviceFlag configured_on;
    const size_t smem = (size_t)(splits > 1 ? Cfg::SMEM_FLOATS : 2 * Cfg::STAGE_FLOATS) * sizeof(float);
    if (!configured_on.here()) {
        if (int32_t s = check_cuda(cudaFuncSetAttribute(matmul_f32_kernel<BM, BN, TRANS_B, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                        (int)(Cfg::SMEM_FLOATS * sizeof(float))), "matmul_f32 smem attr")) return s;
        configured_on.here() = true;
    }
    const int64_t m_tiles = (m + BM - 1) / BM, n_tiles = (n + BN - 1) / BN;
    MFT_CHECK_ARG(m_tiles * n_tiles < (1ll << 31), "mft_matmul_f32: output too large");
    int64_t per = (k + splits - 1) / splits;
    per = (per + BK - 1) / BK * BK;                  // a rank without any K left adds zeros
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(m_tiles * n_tiles), (unsigned)splits, (unsigned)batch);
    cfg.blockDim = dim3(Cfg::THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = (unsigned)splits; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = splits > 1 ? 1 : 0;
    cudaLaunchKernelEx(&cfg, matmul_f32_kernel<BM, BN, TRANS_B, VEC>, a, b, c, (int)m, (int)n, (int)k, (int)n_tiles, (int)per, sa, sb, sc);
    MFT_LAUNCH_CHECK("matmul_f32");
    return MFT_OK;
}

}  // namespace
}  // namespace mft

using namespace mft;

extern "C" int32_t mft_matmul_f32(const float* a, const float* b, float* c, int64_t batch, int64_t m, int64_t n, int64_t k, int64_t stride_a,
                                  int64_t stride_b, int64_t stride_c, int32_t trans_b, mft_stream_t stream) {
    MFT_CHECK_ARG(a && b && c && batch > 0 && m > 0 && n > 0 && k > 0 && batch <= 65535, "mft_matmul_f32: bad argument");
    MFT_CHECK_ARG(m < (1ll << 31) - 128 && n < (1ll << 31) - 128 && k < (1ll << 31) - 128, "mft_matmul_f32: dimension too large");
    const MmPlan p = plan(m, n, k, batch);
    if (small_tiles(m, n, k, batch, trans_b != 0, p)) {
        matmul_f32_small_kernel<<<dim3((unsigned)((n + 31) / 32), (unsigned)((m + 31) / 32), (unsigned)batch), dim3(32, 32), 0, as_stream(stream)>>>(
            a, b, c, (int)m, (int)n, (int)k, stride_a, stride_b, stride_c, trans_b);
        MFT_LAUNCH_CHECK("matmul_f32");
        return MFT_OK;
    }
    // 16-byte accesses need rows that start and end on 16 bytes in all three operands
    auto al = [](const void* q, int64_t stride) { return reinterpret_cast<uintptr_t>(q) % 16 == 0 && stride % 4 == 0; };
    const bool vec = k % 4 == 0 && n % 4 == 0 && al(a, stride_a) && al(b, stride_b) && al(c, stride_c);
    cudaStream_t st = as_stream(stream);
#define MFT_MM(BM, TB, V) launch<BM, BM, TB, V>(a, b, c, batch, m, n, k, stride_a, stride_b, stride_c, p.splits, st)
    if (p.big) return trans_b ? (vec ? MFT_MM(128, true, true) : MFT_MM(128, true, false)) : (vec ? MFT_MM(128, false, true) : MFT_MM(128, false, false));
    return trans_b ? (vec ? MFT_MM(64, true, true) : MFT_MM(64, true, false)) : (vec ? MFT_MM(64, false, true) : MFT_MM(64, false, false));
#undef MFT_MM
}
