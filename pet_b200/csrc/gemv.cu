// Matrix-vector products: C[b,m,n] with m <= 8 rows of A (a classifier head at batch 1, one token against a projection).  The
// 128-row tensor-core tile would be almost empty and the work is one pass over B, so it runs in exact fp32 on the CUDA cores
// and is bound by reading B from HBM.  What that takes: 16-byte loads, eight of them in flight per lane, and CTAs enough to
// keep about 45 KB of loads in flight on every SM: K is split over the CTAs of a thread-block cluster where the columns alone
// are too few, and the partial sums meet in distributed shared memory (added in rank order: no scratch, no second launch).
// 1 x 4096 against 4096 x 4096 (67 MB): 61 us with 4-byte loads and 128 CTAs that each walked all of K behind block-wide
// barriers (1.1 TB/s); this kernel 14.4 us (4.7 TB/s), B as [n][k] 17.5 us, m = 8 against 4096 x 16384 286 -> 80 us.
#include "common.h"
#include "tc_ptx.cuh"
#include <algorithm>

namespace petb200 {

namespace {

constexpr int kGvWarps = 8, kGvThreads = kGvWarps * 32;
// Rows of K whose A values sit in shared memory at a time.
template <int M> constexpr int gemv_tile() { return M <= 4 ? 1024 : 512; }

struct GemvArgs {
    const float *a, *b, *bias, *res;
    float *c;
    int m, n, k, transA, act, ksplit;
};

// K range of this CTA: whole 8-row groups except at the end.
__device__ __forceinline__ void gemv_slice(const GemvArgs &g, int rank, int &k0, int &k1) {
    const int groups = (g.k + 7) / 8;
    k0 = (int)((long long)groups * rank / g.ksplit) * 8;
    k1 = min(g.k, (int)((long long)groups * (rank + 1) / g.ksplit) * 8);
}

// A[.., kt .. kt + kn) into shared memory as sa[row][kk], zero up to the next multiple of PAD (what the product loops read).
template <int M, int PAD>
__device__ __forceinline__ void gemv_load_a(const GemvArgs &g, const float *ab, float (*sa)[gemv_tile<M>()], int kt, int kn) {
    const int kp = (kn + PAD - 1) / PAD * PAD;
    for (int i = threadIdx.x; i < M * kp; i += kGvThreads) {
        const int r = g.transA ? i % M : i / kp, kk = g.transA ? i / M : i - r * kp; // consecutive threads, consecutive addresses
        float v = 0.f;
        if (r < g.m && kk < kn)
            v = __ldg(g.transA ? ab + (long long)(kt + kk) * g.m + r : ab + (long long)r * g.k + kt + kk);
        sa[r][kk] = v;
    }
}

// The CTA's sums of its K slice are in part[row][column]: add up the cluster's and store.  Every thread of every CTA gets here.
template <int M, int COLS>
__device__ __forceinline__ void gemv_finish(const GemvArgs &g, float (*part)[COLS], int col0, int bb, int rank) {
    if (g.ksplit > 1)
        ptx::cluster_sync_all();
    else
        __syncthreads();
    // each rank finishes its share of the block's columns
    const int share = COLS / g.ksplit, c0 = rank * share;
    for (int i = threadIdx.x; i < M * share; i += kGvThreads) {
        const int r = i / share, cl = c0 + i - r * share, col = col0 + cl;
        if (r >= g.m || col >= g.n)
            continue;
        float v = 0.f;
        if (g.ksplit == 1) {
            v = part[r][cl];
        } else {
            const uint32_t at = ptx::smem_u32(&part[r][cl]);
            for (int p = 0; p < g.ksplit; ++p)
                v += ptx::ld_dsmem_f32(ptx::map_to_cta(at, (uint32_t)p));
        }
        if (g.bias)
            v += __ldg(g.bias + col);
        const long long co = ((long long)bb * g.m + r) * g.n + col;
        if (g.res)
            v += __ldg(g.res + co);
        g.c[co] = apply_act(v, g.act);
    }
    if (g.ksplit > 1)
        ptx::cluster_sync_all(); // a CTA's sums stay readable until every peer has read them
}

// B as [k][n]: a lane owns four columns (VEC: adjacent, one 16-byte load; otherwise 32 apart), the warps take alternate groups
// of eight K rows: eight loads in flight per lane.  grid (ceil(n/128), ksplit, batch).
template <int M, bool VEC>
__global__ void __launch_bounds__(kGvThreads, 2) k_gemv_kn(const GemvArgs g) {
    pdl_prologue();
    constexpr int kTile = gemv_tile<M>();
    __shared__ __align__(16) float sa[M][kTile];
    __shared__ float part[M][128];
    __shared__ float red[kGvWarps / 2][M][128];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rank = blockIdx.y, bb = blockIdx.z, col0 = blockIdx.x * 128;
    const float *ab = g.a + (long long)bb * g.m * g.k, *bm = g.b + (long long)bb * g.k * g.n;
    int k0, k1;
    gemv_slice(g, rank, k0, k1);
    float acc[M][4];
#pragma unroll
    for (int r = 0; r < M; ++r)
#pragma unroll
        for (int j = 0; j < 4; ++j)
            acc[r][j] = 0.f;
    constexpr int kStep = kGvWarps * 8;
    const int cl = VEC ? 4 * lane : lane, step = VEC ? 1 : 32;
    bool live[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
        live[j] = col0 + cl + j * step < g.n;
    // eight rows of B, from row kk of the slice on; rows past its end read as zero
    auto fetch = [&](float (&bv)[8][4], int kk) {
        const float *src = bm + (long long)(k0 + kk) * g.n + col0 + cl;
#pragma unroll
        for (int u = 0; u < 8; ++u, src += g.n) {
            const bool in = k0 + kk + u < k1;
            if (VEC) {
                const float4 v = in && live[0] ? __ldg(reinterpret_cast<const float4 *>(src)) : make_float4(0.f, 0.f, 0.f, 0.f);
                bv[u][0] = v.x, bv[u][1] = v.y, bv[u][2] = v.z, bv[u][3] = v.w;
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    bv[u][j] = in && live[j] ? __ldg(src + j * step) : 0.f;
            }
        }
    };
    float b0[8][4], b1[8][4]; // the group being multiplied and the next one, in flight
    fetch(b0, warp * 8);
    for (int kt = 0; kt < k1 - k0; kt += kTile) {
        const int kn = min(kTile, k1 - k0 - kt);
        if (kt > 0)
            __syncthreads(); // the previous tile of A has been consumed
        gemv_load_a<M, 8>(g, ab, sa, k0 + kt, kn);
        __syncthreads();
        auto multiply = [&](const float (&bv)[8][4], int kk) {
#pragma unroll
            for (int r = 0; r < M; ++r) {
                const float4 a0 = *reinterpret_cast<const float4 *>(&sa[r][kk]), a1 = *reinterpret_cast<const float4 *>(&sa[r][kk + 4]);
                const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
                for (int u = 0; u < 8; ++u)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        acc[r][j] = fmaf(av[u], bv[u][j], acc[r][j]);
            }
        };
        for (int kk = warp * 8; kk < kn; kk += 2 * kStep) { // (a tile is a whole number of steps: the groups run on across tiles)
            fetch(b1, kt + kk + kStep);
            multiply(b0, kk);
            fetch(b0, kt + kk + 2 * kStep);
            if (kk + kStep < kn)
                multiply(b1, kk + kStep);
        }
    }
    // the warps' sums, in warp order: the upper half of the warps lays its own down, the lower half adds them in pairs
    if (warp >= kGvWarps / 2)
#pragma unroll
        for (int r = 0; r < M; ++r)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                red[warp - kGvWarps / 2][r][cl + j * step] = acc[r][j];
    __syncthreads();
    if (warp < kGvWarps / 2)
#pragma unroll
        for (int r = 0; r < M; ++r)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                red[warp][r][cl + j * step] += acc[r][j];
    __syncthreads();
    for (int i = threadIdx.x; i < M * 128; i += kGvThreads) {
        const int r = i >> 7, c = i & 127;
        part[r][c] = (red[0][r][c] + red[1][r][c]) + (red[2][r][c] + red[3][r][c]);
    }
    gemv_finish<M, 128>(g, part, col0, bb, rank);
}

// B as [n][k]: a warp owns four columns (rows of B), its lanes split K (VEC: four adjacent values, 16-byte loads) and are added
// up by shuffles.  grid (ceil(n/32), ksplit, batch).
template <int M, bool VEC>
__global__ void __launch_bounds__(kGvThreads, 2) k_gemv_nk(const GemvArgs g) {
    pdl_prologue();
    constexpr int kTile = gemv_tile<M>();
    __shared__ __align__(16) float sa[M][kTile];
    __shared__ float part[M][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rank = blockIdx.y, bb = blockIdx.z, col0 = blockIdx.x * 32;
    const float *ab = g.a + (long long)bb * g.m * g.k, *bm = g.b + (long long)bb * g.k * g.n;
    int k0, k1;
    gemv_slice(g, rank, k0, k1);
    float acc[M][4];
#pragma unroll
    for (int r = 0; r < M; ++r)
#pragma unroll
        for (int j = 0; j < 4; ++j)
            acc[r][j] = 0.f;
    const float *row[4]; // a column past the end reads the last one's row; its sums are never stored
#pragma unroll
    for (int j = 0; j < 4; ++j)
        row[j] = bm + (long long)min(col0 + warp * 4 + j, g.n - 1) * g.k;
    // 128 values of K for each of the four columns, from value kk of the slice on; past its end they read as zero
    auto fetch = [&](float (&bv)[4][4], int kk) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (VEC) { // (slices are whole 8-row groups and k % 4 == 0: a quad is inside or outside)
                const int ke = k0 + kk + lane * 4;
                const float4 v = ke < k1 ? __ldg(reinterpret_cast<const float4 *>(row[j] + ke)) : make_float4(0.f, 0.f, 0.f, 0.f);
                bv[j][0] = v.x, bv[j][1] = v.y, bv[j][2] = v.z, bv[j][3] = v.w;
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int ke = k0 + kk + e * 32 + lane;
                    bv[j][e] = ke < k1 ? __ldg(row[j] + ke) : 0.f;
                }
            }
        }
    };
    float b0[4][4], b1[4][4], b2[4][4], b3[4][4]; // four chunks, multiplied in turn: three to four of them in flight
    fetch(b0, 0), fetch(b1, 128), fetch(b2, 256);
    for (int kt = 0; kt < k1 - k0; kt += kTile) {
        const int kn = min(kTile, k1 - k0 - kt);
        if (kt > 0)
            __syncthreads();
        gemv_load_a<M, 512>(g, ab, sa, k0 + kt, kn);
        __syncthreads();
        auto multiply = [&](const float (&bv)[4][4], int kk) {
#pragma unroll
            for (int r = 0; r < M; ++r) {
                float av[4];
                if (VEC) {
                    const float4 v = *reinterpret_cast<const float4 *>(&sa[r][kk + lane * 4]);
                    av[0] = v.x, av[1] = v.y, av[2] = v.z, av[3] = v.w;
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        av[e] = sa[r][kk + e * 32 + lane];
                }
#pragma unroll
                for (int j = 0; j < 4; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        acc[r][j] = fmaf(av[e], bv[j][e], acc[r][j]);
            }
        };
        for (int kk = 0; kk < kn; kk += 512) { // (A reads as zero up to the next multiple of 512)
            fetch(b3, kt + kk + 384);
            multiply(b0, kk);
            fetch(b0, kt + kk + 512);
            multiply(b1, kk + 128);
            fetch(b1, kt + kk + 640);
            multiply(b2, kk + 256);
            fetch(b2, kt + kk + 768);
            multiply(b3, kk + 384);
        }
    }
#pragma unroll
    for (int r = 0; r < M; ++r)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float v = acc[r][j];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
                v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0)
                part[r][warp * 4 + j] = v;
        }
    gemv_finish<M, 32>(g, part, col0, bb, rank);
}

template <typename K> int gemv_launch(petb200_ctx *ctx, K kern, const GemvArgs &g, dim3 grid, cudaStream_t s) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid, cfg.blockDim = dim3(kGvThreads), cfg.stream = s;
    cudaLaunchAttribute attr[2] = {};
    int n = 0;
    if (g.ksplit > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = 1, attr[n].val.clusterDim.y = (unsigned)g.ksplit, attr[n].val.clusterDim.z = 1;
        ++n;
    }
    if (pdl_enabled()) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    cfg.attrs = attr, cfg.numAttrs = (unsigned)n;
    (void)cudaLaunchKernelEx(&cfg, kern, g); // errors surface through launched()
    return launched(ctx, "k_gemv");
}

template <int M> int gemv_pick(petb200_ctx *ctx, const GemvArgs &g, int transB, dim3 grid, cudaStream_t s) {
    const bool vec = (transB ? g.k : g.n) % 4 == 0 && ((size_t)g.b & 15) == 0; // every row of B starts on 16 bytes
    if (transB)
        return vec ? gemv_launch(ctx, k_gemv_nk<M, true>, g, grid, s) : gemv_launch(ctx, k_gemv_nk<M, false>, g, grid, s);
    return vec ? gemv_launch(ctx, k_gemv_kn<M, true>, g, grid, s) : gemv_launch(ctx, k_gemv_kn<M, false>, g, grid, s);
}

} // namespace

// c = act(op(A) op(B) + bias + res) for m <= 8; a [b][m][k] (or [b][k][m]), b [b][k][n] (or [b][n][k]).
int gemv_run(petb200_ctx *ctx, const float *a, const float *b, const float *bias, const float *res, float *c, int bs, int m, int n, int k,
             int transA, int transB, int act, cudaStream_t s) {
    GemvArgs g{a, b, bias, res, c, m, n, k, transA, act, 1};
    const int cols = transB ? 32 : 128;
    const long long blocks = (long long)((n + cols - 1) / cols) * bs;
    // Split K until there are about two CTAs of 256 threads for every SM (45 KB of loads in flight each SM needs at least
    // that many: 1 x 4096 x 4096 14.4 us = 4.7 TB/s); a CTA keeps at least one pass of its eight warps (64 rows of [k][n], 256 values of a row of [n][k]).
    const int least = transB ? 256 : 64;
    while (g.ksplit < 8 && blocks * g.ksplit < 2LL * ctx->sm_count && k >= 2 * g.ksplit * least)
        g.ksplit *= 2;
    const dim3 grid((unsigned)((n + cols - 1) / cols), (unsigned)g.ksplit, (unsigned)bs);
    if (m <= 1)
        return gemv_pick<1>(ctx, g, transB, grid, s);
    if (m <= 2)
        return gemv_pick<2>(ctx, g, transB, grid, s);
    if (m <= 4)
        return gemv_pick<4>(ctx, g, transB, grid, s);
    return gemv_pick<8>(ctx, g, transB, grid, s);
}

} // namespace petb200
