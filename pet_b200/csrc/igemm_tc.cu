// Plans and launches of the tensor-core kernel (igemm_kernel.cuh): tiling, K split and tensor maps of convolutions, matmuls and
// banded products, and the packing of their B operands.
#include "igemm_kernel.cuh"
#include <algorithm>
#include <array>
#include <map>

namespace petb200 {

// -------------------------------------------------------------------------------------------------------------
// weight packing: W[F][cpg][T] (conv) or B[b][k][n] / B[b][n][k] (matmul) -> hi/lo [rows][Ktot], K ordered as the
// kernel consumes it: k = chunk*Kc_pad + tap*BC + ci, zero where there is no such element.
// -------------------------------------------------------------------------------------------------------------
// hi/lo parts of one packed value: TF32 (hi = top 19 bits, or rounded for a single pass) as fp32 words, or bf16
template <int MATH> __device__ __forceinline__ void store_split(void *hi, void *lo, long long i, float v) {
    if (MATH == kMathBf16x3) {
        const uint32_t h = ptx::pack_bf16x2(v, 0.f) & 0xffffu;
        reinterpret_cast<uint16_t *>(hi)[i] = (uint16_t)h;
        reinterpret_cast<uint16_t *>(lo)[i] = (uint16_t)(ptx::pack_bf16x2(v - __uint_as_float(h << 16), 0.f) & 0xffffu);
    } else {
        const float h = MATH == kMathTf32x1 ? __uint_as_float(ptx::cvt_rna_tf32(v)) : __uint_as_float(__float_as_uint(v) & 0xffffe000u);
        reinterpret_cast<float *>(hi)[i] = h;
        reinterpret_cast<float *>(lo)[i] = v - h;
    }
}

template <int MATH>
__global__ void __launch_bounds__(256) k_pack_conv_w(const float *__restrict__ w, void *__restrict__ hi,
                                                     void *__restrict__ lo, int F, int cpg, int T, int BC, int Kc_pad,
                                                     int nchunks) {
    const long long Ktot = (long long)Kc_pad * nchunks;
    const long long total = (long long)F * Ktot;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const int f = (int)(i / Ktot);
        const int k = (int)(i - (long long)f * Ktot);
        const int ch = k / Kc_pad, kc = k - ch * Kc_pad;
        const int tap = kc / BC, ci = kc - tap * BC;
        const int c = ch * BC + ci;
        float v = 0.f;
        if (tap < T && c < cpg)
            v = __ldg(w + ((long long)f * cpg + c) * T + tap);
        store_split<MATH>(hi, lo, i, v);
    }
}

// Two packed values of fp16, times the filter's factor and unit, in one word of hi and one of lo.
__device__ __forceinline__ void store_halves(void *hi, void *lo, long long word, float a, float b, float factor) {
    a *= factor, b *= factor;
    const uint32_t h = ptx::pack_f16x2(a, b);
    const float2 hf = ptx::unpack_f16x2(h);
    reinterpret_cast<uint32_t *>(hi)[word] = h;
    reinterpret_cast<uint32_t *>(lo)[word] = ptx::pack_f16x2((a - hf.x) * kLoScale, (b - hf.y) * kLoScale);
}
// fp16: a packed filter has a factor (see row_exponent), known only when all of it has been seen.  gridDim.y blocks share filter
// blockIdx.x: each looks at all of it, the second time out of the caches, and packs its part.  (Factors in a launch of their own: 30
// instead of 17 us for the weights of a 512-channel 3x3 layer, call to call, 15 instead of 12 for a 64-channel one.)
struct PackFilters {
    const float *w;
    void *hi, *lo;
    float *unscale;            // what the filter's sums are multiplied by
    uint16_t *numbers, number; // see TcCore::factor_word
    int cpg, T, BC, Ktot;
    FastDiv by_kc_pad, by_bc;
};
__global__ void __launch_bounds__(256) k_pack_conv_f16(const PackFilters g) {
    __shared__ float tops[8];
    const int f = (int)blockIdx.x, lane = threadIdx.x & 31, per_filter = g.cpg * g.T;
    const float *src = g.w + (long long)f * per_filter;
    float top = 0.f;
#pragma unroll 8
    for (int i = threadIdx.x; i < per_filter; i += 256)
        top = fmaxf(top, fabsf(__ldg(src + i)));
    for (int o = 16; o; o >>= 1)
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    if (lane == 0)
        tops[threadIdx.x >> 5] = top;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i)
        top = fmaxf(top, tops[i]);
    const uint32_t e = row_exponent(top);
    const float factor = kFilterUnit / filter_unscale(e);
    if (threadIdx.x == 0 && blockIdx.y == 0) {
        g.unscale[f] = filter_unscale(e);
        if (f == 0)
            g.numbers[0] = g.number;
        if (filter_out_of_range(e))
            g.numbers[1] = g.number;
    }
    auto at = [&](int k) { // value at a packed position: 0 past the taps of a chunk or the channels of the filter
        const int ch = g.by_kc_pad.div(k), kc = k - ch * (int)g.by_kc_pad.d, tap = g.by_bc.div(kc), c = ch * g.BC + kc - tap * g.BC;
        return tap < g.T && c < g.cpg ? __ldg(src + c * g.T + tap) : 0.f;
    };
    const int words = g.Ktot / 2; // (a multiple of 32: whole stages of 64)
#pragma unroll 4
    for (int i = (int)blockIdx.y * 256 + threadIdx.x; i < words; i += (int)gridDim.y * 256)
        store_halves(g.hi, g.lo, (long long)f * words + i, at(2 * i), at(2 * i + 1), factor);
}

// What a matmul needs before it can run, in one launch (bound by HBM: every operand read once, its copy written once).
// Blocks [0, b_tiles): B[b][k][n] or [b][n][k] -> hi/lo [rows][Kpad], a tile of 32 rows x 32 packed positions per block; a [k][n]
// tile is turned through shared memory, so that both sides move whole 128-byte lines (one thread per packed position read B
// with a stride of n words: 35 us of the 76 us of a 4 x 500 x 1001 x 770 product).  The other blocks: rows of A copied to a
// pitch that TMA can address (the padding is zero).
struct PrepareArgs {
    const float *b;
    void *hi, *lo;
    int bs, n, k, Kpad, BC;
    float *unscale;          // fp16: what the sums of each packed row are multiplied by
    uint16_t *numbers, number; // see TcCore::factor_word
    FastDiv by_kc_pad, by_tiles_k, by_tiles_n;
    long long sb_batch, sb_row;
    int b_tiles, tiles_k, tiles_n;
    int split;              // fp16: CTAs per strip of columns (a cluster) or warps per row, a power of two
    const float *a;
    float *a_copy;
    long long a_rows;
    int a_w, a_pitch;
};
// Rows of A, a warp each; `block` of the launch's `blocks` that do this.
__device__ __forceinline__ void copy_a_rows(const PrepareArgs &g, int block, int blocks) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (long long r = (long long)block * 8 + warp; r < g.a_rows; r += (long long)blocks * 8) {
        const float *src = g.a + r * g.a_w;
        float *dst = g.a_copy + r * g.a_pitch;
#pragma unroll 8
        for (int c = lane; c < g.a_pitch; c += 32)
            dst[c] = c < g.a_w ? __ldg(src + c) : 0.f;
    }
}
template <int MATH, bool TRANSB>
__global__ void __launch_bounds__(256) k_prepare_mm(const PrepareArgs g) {
    pdl_prologue();
    __shared__ float tile[32][33];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if ((int)blockIdx.x >= g.b_tiles) {
        copy_a_rows(g, (int)blockIdx.x - g.b_tiles, (int)gridDim.x - g.b_tiles);
        return;
    }
    const int rest = g.by_tiles_k.div((int)blockIdx.x), tk = (int)blockIdx.x - rest * g.tiles_k, bb = g.by_tiles_n.div(rest), tn = rest - bb * g.tiles_n;
    const float *src = g.b + bb * g.sb_batch;
    const int k0 = tk * 32, n0 = tn * 32;
    // packed position -> row of B: chunk * Kc_pad + element of the chunk (BC of them, then padding; Kc_pad a multiple of 32)
    const int ch = g.by_kc_pad.div(k0), kc0 = k0 - ch * (int)g.by_kc_pad.d, kk0 = ch * g.BC + kc0, kn = min(min(g.BC - kc0, g.k - kk0), 32);
    if constexpr (TRANSB) {
#pragma unroll
        for (int i = 0; i < 32; i += 8) {
            const int nn = n0 + warp + i;
            const float v = lane < kn && nn < g.n ? __ldg(src + nn * g.sb_row + kk0 + lane) : 0.f;
            if (nn < g.n)
                store_split<MATH>(g.hi, g.lo, ((long long)bb * g.n + nn) * g.Kpad + k0 + lane, v);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 32; i += 8)
            tile[warp + i][lane] = warp + i < kn && n0 + lane < g.n ? __ldg(src + (kk0 + warp + i) * g.sb_row + n0 + lane) : 0.f;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 32; i += 8) {
            const int nn = n0 + warp + i;
            if (nn < g.n)
                store_split<MATH>(g.hi, g.lo, ((long long)bb * g.n + nn) * g.Kpad + k0 + lane, tile[lane][warp + i]);
        }
    }
}

// The same for fp16, where a packed row (a column of B) has one factor, known only when all of it has been seen (row_exponent).
// Both kernels read B once from memory and write each packed word once, 128 bytes per warp.
// B[b][k][n]: the CTAs of a cluster share a strip of W columns, each a range of 64-position units of the packed row; the units
// stay in shared memory (as many as there is room for, more are read again) while the columns' maxima meet through the cluster.
// W = 8 where strips of 32 would leave SMs idle (3 x 3960 x 36: 8.0 -> 5.0 us, the packing for TF32 takes 3.1).
constexpr int kPrepUnit = 64, kPrepKeep = 8;
template <int W> constexpr int kPrepPitch = W + 1;
template <int W> constexpr int kPrepRoom = W == 32 ? kPrepKeep : 24; // units
template <int W> constexpr size_t kPrepSmem = (size_t)kPrepRoom<W> * kPrepUnit *kPrepPitch<W> * 4;
// Unit u of the packed row: first row of B, number of rows.
__device__ __forceinline__ void prep_unit(const PrepareArgs &g, int u, int &kk0, int &kn) {
    const int k0 = u * kPrepUnit, ch = g.by_kc_pad.div(k0), kc0 = k0 - ch * (int)g.by_kc_pad.d;
    kk0 = ch * g.BC + kc0;
    kn = min(min(g.BC - kc0, g.k - kk0), kPrepUnit);
}
template <int W> __global__ void __launch_bounds__(256) k_prepare_f16_kn(const PrepareArgs g) {
    pdl_prologue();
    constexpr int kPitch = kPrepPitch<W>, kRoom = kPrepRoom<W>, kRows = 32 / W /*of a load*/, kLoads = kPrepUnit / (8 * kRows);
    extern __shared__ float keep[]; // [unit][row][kPitch]
    __shared__ float tops[8][32], column_top[W], factor[W];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, col = lane & (W - 1), row0 = warp * kRows + lane / W;
    if ((int)blockIdx.x >= g.b_tiles) {
        copy_a_rows(g, (int)blockIdx.x - g.b_tiles, (int)gridDim.x - g.b_tiles);
        return; // (whole clusters: b_tiles is a multiple of the cluster)
    }
    const int rank = (int)blockIdx.x % g.split, strip = (int)blockIdx.x / g.split, bb = g.by_tiles_n.div(strip), n0 = (strip - bb * g.tiles_n) * W;
    const int u0 = rank * g.tiles_k / g.split, u1 = (rank + 1) * g.tiles_k / g.split;
    const float *src = g.b + bb * g.sb_batch + n0 + col;
    const bool col_ok = n0 + col < g.n;
    float top = 0.f;
    auto load = [&](int u, float *dst) { // 64 rows of the strip to shared memory
        int kk0, kn;
        prep_unit(g, u, kk0, kn);
        float v[kLoads];
#pragma unroll
        for (int i = 0; i < kLoads; ++i) {
            const int r = row0 + 8 * kRows * i;
            v[i] = col_ok && r < kn ? __ldg(src + (kk0 + r) * g.sb_row) : 0.f;
        }
#pragma unroll
        for (int i = 0; i < kLoads; ++i) {
            top = fmaxf(top, fabsf(v[i]));
            dst[(row0 + 8 * kRows * i) * kPitch + col] = v[i];
        }
    };
#pragma unroll (W == 32 ? 2 : 4)
    for (int u = u0; u < u1; ++u) // units beyond the room take turns in the last place: their maxima count, they are read again
        load(u, keep + min(u - u0, kRoom - 1) * kPrepUnit * kPitch);
#pragma unroll
    for (int o = W; o < 32; o *= 2)
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    tops[warp][lane] = top;
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int i = 1; i < 8; ++i)
            top = fmaxf(top, tops[i][lane]);
        if (lane < W)
            column_top[lane] = top;
    }
    if (g.split > 1) {
        ptx::cluster_sync_all();
        if (warp == 0)
            for (int r = 0; r < g.split; ++r)
                top = fmaxf(top, ptx::ld_dsmem_f32(ptx::map_to_cta(ptx::smem_u32(column_top + col), (uint32_t)r)));
        ptx::cluster_arrive(); // (waited for at the end: nobody leaves while its maxima are being read)
    }
    if (warp == 0 && lane < W) {
        const uint32_t e = row_exponent(top);
        factor[lane] = kFilterUnit / filter_unscale(e);
        if (rank == 0 && col_ok) {
            g.unscale[(long long)bb * g.n + n0 + lane] = filter_unscale(e);
            if (blockIdx.x == 0 && lane == 0)
                g.numbers[0] = g.number;
            if (filter_out_of_range(e))
                g.numbers[1] = g.number;
        }
    }
    __syncthreads();
#pragma unroll 2
    for (int u = u0; u < u1; ++u) {
        const int slot = min(u - u0, kRoom - 1);
        const float *tile = keep + slot * kPrepUnit * kPitch;
        if (u1 - u0 > kRoom && u - u0 >= kRoom - 1) {
            __syncthreads();
            load(u, keep + slot * kPrepUnit * kPitch);
            __syncthreads();
        }
#pragma unroll
        for (int c = warp; c < W; c += 8)
            if (n0 + c < g.n)
                store_halves(g.hi, g.lo, (((long long)bb * g.n + n0 + c) * g.Kpad + u * kPrepUnit) / 2 + lane, tile[2 * lane * kPitch + c],
                             tile[(2 * lane + 1) * kPitch + c], factor[c]);
    }
    if (g.split > 1)
        ptx::cluster_wait();
}
// B[b][n][k]: a packed row is a row of B; g.split warps share it.  A warp keeps its first KEEP units in registers, all loads in
// flight at once; more are read a second time.  (All of them twice, a warp to a row where there were many rows: 29 x 140 rows of 3476 66 us,
// now 27, 4096 of 4096 97, now 40, 4 x 1001 of 770 12.4, now 7.5; the packing for TF32 44, 50, 7.6.)
template <int KEEP> __global__ void __launch_bounds__(256) k_prepare_f16_nk(const PrepareArgs g) {
    pdl_prologue();
    __shared__ float tops[8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if ((int)blockIdx.x >= g.b_tiles) {
        copy_a_rows(g, (int)blockIdx.x - g.b_tiles, (int)gridDim.x - g.b_tiles);
        return;
    }
    const int step = g.split, u0 = warp & (step - 1); // (a power of two)
    const long long row = (long long)blockIdx.x * (8 / step) + warp / step;
    const bool row_ok = row < (long long)g.bs * g.n;
    const int u1 = row_ok ? g.tiles_k : 0;
    const int bb = row_ok ? (int)(row / g.n) : 0, nn = row_ok ? (int)(row - (long long)bb * g.n) : 0;
    const float *src = g.b + bb * g.sb_batch + nn * g.sb_row;
    auto take = [&](int u) {
        int kk0, kn;
        prep_unit(g, u, kk0, kn);
        return make_float2(2 * lane < kn ? __ldg(src + kk0 + 2 * lane) : 0.f, 2 * lane + 1 < kn ? __ldg(src + kk0 + 2 * lane + 1) : 0.f);
    };
    float2 v[KEEP];
#pragma unroll
    for (int i = 0; i < KEEP; ++i)
        v[i] = u0 + i * step < u1 ? take(u0 + i * step) : make_float2(0.f, 0.f);
    float top = 0.f;
#pragma unroll 4
    for (int u = u0 + KEEP * step; u < u1; u += step) {
        const float2 x = take(u);
        top = ptx::max3_abs(top, x.x, x.y);
    }
#pragma unroll
    for (int i = 0; i < KEEP; ++i)
        top = ptx::max3_abs(top, v[i].x, v[i].y);
    for (int o = 16; o; o >>= 1)
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    if (step > 1) {
        if (lane == 0)
            tops[warp] = top;
        __syncthreads();
        for (int i = 0; i < step; ++i)
            top = fmaxf(top, tops[(warp & ~(step - 1)) + i]);
    }
    const uint32_t e = row_exponent(top);
    const float factor = kFilterUnit / filter_unscale(e);
    if (row_ok && u0 == 0 && lane == 0) {
        g.unscale[row] = filter_unscale(e);
        if (row == 0)
            g.numbers[0] = g.number;
        if (filter_out_of_range(e))
            g.numbers[1] = g.number;
    }
    auto put = [&](int u, float2 x) { store_halves(g.hi, g.lo, (row * g.Kpad + u * kPrepUnit) / 2 + lane, x.x, x.y, factor); };
#pragma unroll
    for (int i = 0; i < KEEP; ++i)
        if (u0 + i * step < u1)
            put(u0 + i * step, v[i]);
#pragma unroll 4
    for (int u = u0 + KEEP * step; u < u1; u += step)
        put(u, take(u));
}

// -------------------------------------------------------------------------------------------------------------
// host side
// -------------------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    }
    return fn;
}

static int env_int_early(const char *name, int dflt) {
    const char *v = getenv(name);
    return v ? atoi(v) : dflt;
}

struct TcCore {
    int beside = 1; // launches of this size that share the GPU (a split of K then only adds work)
    petb200_ctx *ctx = nullptr;
    IgemmParams P{};
    int math = kMathTf32x3; // the kernel's PASSES
    bool half() const { return math == kMathBf16x3 || math == kMathF16x3; } // 16-bit operands: 64 K elements per stage
    dim3 grid;
    size_t smem = 0;
    // geometry needed to (re)encode the activation map
    int xd[5]{}; // W,H,D,C,N of the activation tensor as the kernel sees it
    long long a_row = 0, a_batch = 0; // row-major matmul A: element strides of a row and of a batch entry
    long long Ktot = 0;
    int rows_b = 0;
    DevBuf whi, wlo, koff;
    std::vector<int> offsets; // what `koff` holds: made by the configuration (of which a plan may go through two), uploaded once
    // fp16: a factor per packed row of B, and behind them a word of two halves: the number of the last packing (modulo 2^16), and that
    // of the last one which found a factor other than 1.  The kernel multiplies where they are equal.  Both are written by the
    // packing and read by the product on the device: a launch that a CUDA graph holds is replayed after packings that came later
    // than its capture.  (An old number in the second half may come round again, or a graph repeat its own packing: the sums are
    // then multiplied by ones.)  One word and not two: a second register kept through the transform loop cost 0.15 to 0.4 us a
    // launch.  A plan that borrows another's operand has `packed_by` point there.
    DevBuf fscale_buf;
    uint16_t packings = 0;
    const TcCore *packed_by = nullptr;
    uint32_t *factor_word() const { return (uint32_t *)fscale_buf.p + rows_b; }
    long long y_elems = 0;
    CUtensorMap map_x{}, map_bhi{}, map_blo{};
    const void *map_x_ptr = nullptr;
    bool weights_ready = false;
    bool finished = false; // P's derived members are there
    int starve = 0;

    KernelFn kernel() const {
        const int pp = !P.pp ? kSingle : (P.BN <= 64 && P.fl == 0 ? kNarrow : kWide);
        if (P.a_kmajor && P.band_w > 0) // banded products: G2BMM in persistent mode with its own epilogue, GBMML with its own operand fetch
            return igemm_band(P.band_g2 ? 1 : 2, pp);
        switch (math) {
        case kMathTf32x1: return igemm_tf32x1(P.a_kmajor, pp);
        case kMathBf16x3: return igemm_bf16x3(P.a_kmajor, pp);
        case kMathF16x3: return igemm_f16x3(P.a_kmajor, pp);
        default: return igemm_tf32x3(P.a_kmajor, pp);
        }
    }
    int encode_x(const float *x) {
        if (x == map_x_ptr)
            return PETB200_OK;
        EncodeTiledFn enc = encode_fn();
        if (!enc)
            return fail(ctx, PETB200_ERR_CUDA, "cuTensorMapEncodeTiled entry point unavailable");
        if (P.a_kmajor) { // A[b][m][k] row-major: dims (k, m, b), one 128B-swizzled [128 rows][32 k] box per K stage
            cuuint64_t d3[3] = {(cuuint64_t)xd[0], (cuuint64_t)xd[1], (cuuint64_t)xd[2]};
            cuuint64_t s3[2] = {(cuuint64_t)a_row * 4, (cuuint64_t)a_batch * 4};
            cuuint32_t b3[3] = {(cuuint32_t)kStageK, (cuuint32_t)kTileM, 1};
            cuuint32_t e3[3] = {1, 1, 1};
            CUresult r3 = enc(&map_x, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float *>(x), d3, s3, b3, e3,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
            if (r3 != CUDA_SUCCESS)
                return fail(ctx, PETB200_ERR_CUDA, "cuTensorMapEncodeTiled(row-major A) failed with %d", (int)r3);
            map_x_ptr = x;
            return PETB200_OK;
        }
        if (P.flat) { // each image is one run of C*D*H*W floats, viewed as rows of flat_w
            const cuuint64_t run = (cuuint64_t)xd[0] * xd[1] * xd[2] * xd[3];
            cuuint64_t d3[3] = {(cuuint64_t)P.flat_w, run / P.flat_w, (cuuint64_t)xd[4]};
            cuuint64_t s3[2] = {(cuuint64_t)P.flat_w * 4, run * 4};
            cuuint32_t b3[3] = {(cuuint32_t)P.flat_w, (cuuint32_t)P.flat_rows, (cuuint32_t)P.RN};
            cuuint32_t e3[3] = {1, 1, 1};
            CUresult r3 = enc(&map_x, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float *>(x), d3, s3, b3, e3,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
            if (r3 != CUDA_SUCCESS)
                return fail(ctx, PETB200_ERR_CUDA, "cuTensorMapEncodeTiled(flat activations) failed with %d", (int)r3);
            map_x_ptr = x;
            return PETB200_OK;
        }
        cuuint64_t dims[5] = {(cuuint64_t)xd[0], (cuuint64_t)xd[1], (cuuint64_t)xd[2], (cuuint64_t)xd[3], (cuuint64_t)xd[4]};
        cuuint64_t str[4] = {(cuuint64_t)xd[0] * 4, (cuuint64_t)xd[0] * xd[1] * 4, (cuuint64_t)xd[0] * xd[1] * xd[2] * 4,
                             (cuuint64_t)xd[0] * xd[1] * xd[2] * xd[3] * 4};
        cuuint32_t box[5] = {(cuuint32_t)P.RW, (cuuint32_t)P.RH, (cuuint32_t)P.RD, (cuuint32_t)P.BC, (cuuint32_t)P.RN};
        cuuint32_t es[5] = {1, 1, 1, 1, 1};
        CUresult r = enc(&map_x, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 5, const_cast<float *>(x), dims, str, box, es,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS)
            return fail(ctx, PETB200_ERR_CUDA, "cuTensorMapEncodeTiled(activations) failed with %d", (int)r);
        map_x_ptr = x;
        return PETB200_OK;
    }
    int upload_offsets() {
        if (koff.alloc(offsets.size() * 4) != cudaSuccess)
            return fail(ctx, PETB200_ERR_NOMEM, "koff allocation failed");
        PETB200_CUDA(ctx, cudaMemcpy(koff.p, offsets.data(), offsets.size() * 4, cudaMemcpyHostToDevice));
        return PETB200_OK;
    }
    int alloc_b() { // the packed operand: rows_b rows of Ktot elements, hi and lo
        if (int rc = upload_offsets())
            return rc;
        const size_t bytes = (size_t)rows_b * Ktot * (half() ? 2 : 4);
        if (whi.alloc(bytes) != cudaSuccess || wlo.alloc(bytes) != cudaSuccess || (P.f16 && fscale_buf.alloc((size_t)(rows_b + 1) * 4) != cudaSuccess))
            return fail(ctx, PETB200_ERR_NOMEM, "packed operand allocation (%zu bytes) failed", 2 * bytes);
        return encode_b();
    }
    int encode_b() {
        EncodeTiledFn enc = encode_fn();
        if (!enc)
            return fail(ctx, PETB200_ERR_CUDA, "cuTensorMapEncodeTiled entry point unavailable");
        cuuint64_t dims[2] = {(cuuint64_t)Ktot, (cuuint64_t)rows_b};
        cuuint64_t str[1] = {(cuuint64_t)Ktot * (half() ? 2 : 4)};
        cuuint32_t box[2] = {(cuuint32_t)P.ke, (cuuint32_t)P.BN}; // one 128-byte row of K per filter
        cuuint32_t es[2] = {1, 1};
        for (int i = 0; i < 2; ++i) {
            CUresult r = enc(i ? &map_blo : &map_bhi, half() ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2,
                             i ? wlo.p : whi.p, dims, str, box,
                             es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
            if (r != CUDA_SUCCESS)
                return fail(ctx, PETB200_ERR_CUDA, "cuTensorMapEncodeTiled(weights) failed with %d", (int)r);
        }
        return PETB200_OK;
    }
    int launch(const float *x, const float *bias, const float *res, float *y, cudaStream_t s, int link = 0) {
        int rc = encode_x(x);
        if (rc)
            return rc;
        if (!finished) {
            finish_params(P, grid.x);
            finished = true;
        }
        IgemmParams p = P;
        p.link = link;
        p.bias = bias;
        p.res = res;
        p.y = y;
        p.koff = (const int *)koff.p;
        if (P.f16) {
            const TcCore *o = packed_by ? packed_by : this;
            p.fscale = (const float *)o->fscale_buf.p, p.factor_word = o->factor_word();
        }
        p.status = ctx->d_status;
        p.starve = starve;
        p.has_bias = (P.has_bias && bias) ? 1 : 0;
        KernelFn kern = kernel();
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = grid;
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = s;
        cudaLaunchAttribute attr[2] = {};
        int nattr = 0;
        if (P.ksplit > 8 && cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
            (void)cudaGetLastError();
            return fail(ctx, PETB200_ERR_UNSUPPORTED, "clusters of %d CTAs are not allowed on this device", P.ksplit);
        }
        if (P.ksplit > 1) { // the splits of one output tile are consecutive in blockIdx.y: one cluster
            attr[nattr].id = cudaLaunchAttributeClusterDimension;
            attr[nattr].val.clusterDim.x = 1;
            attr[nattr].val.clusterDim.y = (unsigned)P.ksplit;
            attr[nattr].val.clusterDim.z = 1;
            ++nattr;
        }
        if (pdl_enabled()) { // this kernel's set-up may overlap the end of the kernel before it in the stream
            attr[nattr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[nattr].val.programmaticStreamSerializationAllowed = 1;
            ++nattr;
        }
        cfg.attrs = nattr ? attr : nullptr;
        cfg.numAttrs = (unsigned)nattr;
        cudaError_t le = cudaLaunchKernelEx(&cfg, kern, map_x, map_bhi, map_blo, p);
        if (le != cudaSuccess) {
            (void)cudaGetLastError();
            return fail(ctx, PETB200_ERR_CUDA, "launch of k_igemm failed: %s", cudaGetErrorString(le));
        }
        return launched(ctx, "k_igemm");
    }
};

// Geometry of the convolution as the tensor-core kernel sees it.
struct ConvGeom {
    int N, C, D, H, W, Wst /*row pitch of the stored tensor, >= W*/, F, T3[3] /*t,r,s*/, pad[3], stride[3], dil[3], groups;
    int OD, OH, OW;
};

static int env_int(const char *name, int dflt) {
    const char *v = getenv(name);
    return v ? atoi(v) : dflt;
}

// How many clusters of `ks` CTAs of this kernel (one CTA per SM) the device can hold at once: asked of the driver once
// per size (clusters stay inside a GPC, which leaves some SMs of every GPC without a cluster).
static int cluster_slots(petb200_ctx *ctx, int ks) {
    const int sm_count = ctx->sm_count;
    if (ks <= 1)
        return sm_count;
    if (ctx->cluster_slots[ks] == 0) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(1, (unsigned)ks * 64, 1);
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = 200 * 1024; // enough that two CTAs never share an SM, as in every real plan
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 1, attr[0].val.clusterDim.y = (unsigned)ks, attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr, cfg.numAttrs = 1;
        int n = 0;
        (void)cudaFuncSetAttribute(igemm_f16x3(false, kSingle), cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (ks > 8) // clusters of 16 are beyond the portable size: allowed per function
            (void)cudaFuncSetAttribute(igemm_f16x3(false, kSingle), cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (cudaOccupancyMaxActiveClusters(&n, igemm_f16x3(false, kSingle), &cfg) != cudaSuccess || n <= 0) {
            (void)cudaGetLastError();
            // what B200 was measured to hold; a cluster of 16 is only used where the driver itself says it fits
            n = ks > 8 ? -1 : std::max(1, (sm_count * (ks <= 2 ? 96 : 86) / 100) / ks);
        }
        ctx->cluster_slots[ks] = n;
    }
    return ctx->cluster_slots[ks];
}

// Rough cycle model of one launch, used to pick the tile width and the K split.  All constants are measured on row-major products of
// 16 to 1000 rows with every width and split forced in turn: start-up to the first MMA 6300; a K stage 570 / 655 / 890 at 32 /
// 64 / 128 filters (3xTF32, 32 K) and 910 / 910 / 1045 (halves, 64 K); the epilogue of an unsplit tile 34 a filter; the exchange
// through a cluster, reduction and stores together 2300 / 2500 / 8000 and 70 a filter of the CTA's share, which makes a split of a
// 128-filter tile in two the dearest (12500).  Several unsplit tiles in turn hide start-up and epilogue (persistent tiles).
// Against the fastest of all pairs on 57 shapes (these products, ResNet layers at batch 1 to 16): within 2 % on 54; the others lose
// 4, 11 and 14 % (64 x 1000 x 256, a 200-channel 3x3 at 3 x 20 x 20, 16 x 3072 x 768).  The constants before lost up to 31 % on 12 of them.
//   A convolution whose stages each need a raw tile of their own takes 1000 a stage whatever its width (328 channels of 1x1 in chunks
// of 8 to 511 filters: BN 64 26.4 us, BN 128 with K split in two 21.0). A long activation adds 42 a filter, twice that in persistent
// tiles, which four warps store and not eight (768 x 89 x 873, three times, with GELU: 20.3 us in tiles of 64, 17.9 in 128).
// A filter of a persistent tile's epilogue costs twice that of another's for the same reason (8 x 29 x 51 x 1454: 13.4 us in tiles of 32, 11.9
// in 128).  `beside`: launches that share the GPU, none of which is persistent.
static double est_cycles(petb200_ctx *ctx, long long ctas, const IgemmParams &P, int math, int ks, int beside) {
    const int BN = P.BN, w = BN <= 32 ? 0 : (BN <= 64 ? 1 : 2);
    static const double tf32[3] = {570, 655, 890}, halves[3] = {910, 910, 1045}, exchange[3] = {2300, 2500, 8000};
    const double mma = math == kMathTf32x1 ? 520.0 : (math == kMathTf32x3 ? tf32[w] : halves[w]), start = 6300.0;
    const double gather = !P.a_kmajor && P.spc == 1 ? 1000.0 : 0.0;
    const double stages = (double)((P.nchunks + ks - 1) / ks) * P.spc, stage = std::max(mma, gather);
    const long long slots = cluster_slots(ctx, ks);
    if (slots <= 0)
        return 1e30; // this cluster size cannot be launched here
    const bool long_act = P.act > PETB200_ACT_RELU;
    const double waves = (double)((ctas * beside + slots - 1) / slots), filters = (double)P.Fg / ((P.Fg + BN - 1) / BN);
    const double epilogue = (34.0 + (long_act ? 42.0 : 0.0)) * filters * (waves > 1 && beside == 1 ? 2.0 : 1.0);
    if (ks > 1)
        return waves * (start + stages * stage + exchange[w] + (70.0 + (long_act ? 42.0 : 0.0)) * BN / ks);
    return start + waves * std::max(stages * stage, epilogue) + (waves - 1) * 1200.0 + epilogue;
}
// Split K over 1, 2, 4, 8 or 16 CTAs (a cluster; 16 is beyond the portable cluster size and allowed per function): the
// split must divide the tile width and leave every CTA a chunk.
static int choose_ksplit(petb200_ctx *ctx, long long ctas, const IgemmParams &P, int math, int want, int beside, double *cycles) {
    auto ok = [&](int ks) { return ks == 1 || (ks <= P.nchunks && P.BN % ks == 0); };
    int best = 1;
    double best_c = est_cycles(ctx, ctas, P, math, 1, beside);
    static const int ks_cap = std::min(16, std::max(1, env_int_early("PETB200_TC_KSPLIT_MAX", 16)));
    if (want > 0) {
        for (best = 16; best > 1 && !(best <= want && ok(best) && cluster_slots(ctx, best) > 0); best /= 2) {
        }
        best_c = est_cycles(ctx, ctas, P, math, best, beside);
    } else {
        for (int ks = 2; ks <= ks_cap; ks *= 2) {
            if (!ok(ks))
                continue;
            const double c = est_cycles(ctx, ctas, P, math, ks, beside);
            if (c < best_c * 0.97) // a deeper split has to pay for itself
                best = ks, best_c = c;
        }
    }
    if (cycles)
        *cycles = best_c;
    return best;
}

// Accumulator flush period (see IgemmParams::fl).  The truncation bias of the tensor core's fp32 accumulator grows with the number
// of MMAs added into one running sum: K ranges of more than `3 * period` stages per CTA are drained every `period` stages
// (PETB200_TC_FLUSH in the environment, 0 = never; measured without a flush: 2.4e-4 of the contract's 1e-3 at 18 stages,
// 3e-4..4e-4 at 36, 2e-3 at 54).
static void choose_flush(TcCore &core) {
    IgemmParams &P = core.P;
    // (bf16: twice the K per stage and an accuracy class that the split, not the truncation, dominates: half as often.  fp16: a stage
    // is 64 K in four MMAs per accumulator, half the truncations of TF32 for the same K; both go without up to K = 768, where
    // 384 x 3072 x 768 shows 9.5e-7 of the exact result's norm against 1.7e-6, and beyond it 4 x 500 x 1001 x 770 was at 9.8e-7
    // unflushed against TF32's flushed 9.1e-7)
    const int period = env_int("PETB200_TC_FLUSH", core.math == kMathBf16x3 ? 16 : 8);
    const int ks_max = ((P.nchunks + P.ksplit - 1) / P.ksplit) * P.spc, unflushed = core.math == kMathF16x3 ? 3 * period / 2 : 3 * period;
    P.fl = (core.math != kMathTf32x1 && period > 0 && ks_max > unflushed) ? period : 0;
    if (env_int("PETB200_TC_VERBOSE", 0))
        fprintf(stderr, "[petb200] igemm plan: BN %d BC %d chunks %d stages/chunk %d ksplit %d flush %d NB %d NR %d kmajor %d flat %d math %s\n",
                P.BN, P.BC, P.nchunks, P.spc, P.ksplit, P.fl, P.NB, P.NR, P.a_kmajor, P.flat,
                core.math == kMathTf32x1 ? "1xtf32" : (core.math == kMathBf16x3 ? "bf16x3" : (core.math == kMathF16x3 ? "f16x3" : "3xtf32")));
}

// Persistent mode (see IgemmParams::pp) where some SM would otherwise run several CTAs in sequence: the start-up of a CTA (see
// est_cycles) and its epilogue hide behind the MMAs of its neighbour tiles.  Not with a K
// split (a CTA's tile is then a cluster's).  Sets the grid.
static void choose_grid(petb200_ctx *ctx, TcCore &core, int mtiles, int ntiles, int gz, size_t budget) {
    IgemmParams &P = core.P;
    const long long tiles = (long long)mtiles * ntiles * gz;
    P.mtiles = mtiles, P.ntiles = ntiles, P.tiles = (int)tiles;
    P.pp = 0;
    core.grid = dim3((unsigned)mtiles, (unsigned)(ntiles * P.ksplit), (unsigned)gz);
    if (!env_int("PETB200_TC_PINGPONG", 1) || P.ksplit > 1 || tiles <= ctx->sm_count || tiles > (1 << 30))
        return;
    const int nb_was = P.NB, nr_was = P.NR;
    P.pp = 1;
    while (smem_layout(P).total > budget && (P.NB > 2 || P.NR > 2)) // the drain warps' blocks take room from the rings
        (P.NB > 2 && P.NB >= P.NR ? P.NB : P.NR)--;
    if (smem_layout(P).total > budget) {
        P.pp = 0, P.NB = nb_was, P.NR = nr_was;
        return;
    }
    const long long per_cta = (tiles + ctx->sm_count - 1) / ctx->sm_count;
    core.grid = dim3((unsigned)((tiles + per_cta - 1) / per_cta), 1, 1);
}

// The dynamic shared-memory attribute is per function and device, not per launch: each context raises it once to the device limit
// so that plans with different needs can coexist.
static int raise_smem_limit(petb200_ctx *ctx) {
    if (ctx->tc_attr_set)
        return PETB200_OK;
    const int lim = (int)std::min<size_t>(ctx->smem_optin, 227 * 1024);
    cudaError_t e = cudaSuccess;
    auto raise = [&](KernelFn k) {
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
    };
    for (int pp : {(int)kSingle, (int)kNarrow, (int)kWide}) {
        for (auto family : {igemm_tf32x3, igemm_f16x3, igemm_tf32x1, igemm_bf16x3})
            raise(family(false, pp)), raise(family(true, pp));
        raise(igemm_band(2, pp));
    }
    raise(igemm_band(1, kNarrow));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_prepare_f16_kn<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPrepSmem<32>);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_prepare_f16_kn<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPrepSmem<8>);
    if (e != cudaSuccess)
        return fail(ctx, PETB200_ERR_CUDA, "cudaFuncSetAttribute(%d bytes) failed: %s", lim, cudaGetErrorString(e));
    ctx->tc_attr_set = true;
    return PETB200_OK;
}

// Fills core.P (tiling, raw box, stage counts) for a window [oh0,ohn) x [ow0,own) of the output; returns
// PETB200_ERR_UNSUPPORTED when the shape does not fit this kernel's constraints.
static int tc_configure(petb200_ctx *ctx, TcCore &core, const ConvGeom &g, int oh0, int ohn, int ow0, int own,
                        int z_is_batch, int images, long long ys_n, long long ys_f, long long ys_p, int has_bias, int act,
                        int force_bc = 0, int force_ksplit = 0, int force_bn = 0, int flat = 0, int max_ipt = 0) {
    IgemmParams &P = core.P;
    const int cpg = g.C / g.groups, Fg = g.F / g.groups;
    if (!flat && g.Wst % 4 != 0)
        return fail(ctx, PETB200_ERR_UNSUPPORTED, "the TMA box needs a row pitch divisible by 4, got %d", g.Wst);
    P.flat = flat ? 1 : 0;
    P.ke = core.half() ? 64 : kStageK;
    P.f16 = core.math == kMathF16x3;
    P.xD = g.D, P.xH = g.H, P.xW = g.W;
    for (int i = 0; i < 3; ++i)
        P.T3[i] = g.T3[i], P.dil[i] = g.dil[i];
    P.OD = g.OD;
    P.OH = g.OH;
    P.OW = g.OW;
    P.oh0 = oh0;
    P.ohn = ohn;
    P.ow0 = ow0;
    P.own = own;
    P.Pw = ohn * own;
    P.units = (z_is_batch ? 1 : images) * g.OD;
    P.sd = g.stride[0];
    P.sh = g.stride[1];
    P.sw = g.stride[2];
    P.pd = g.pad[0];
    P.ph = g.pad[1];
    P.pw = g.pad[2];
    P.cpg = cpg;
    P.Fg = Fg;
    P.z_is_batch = z_is_batch;
    P.ys_n = ys_n;
    P.ys_f = ys_f;
    P.ys_p = ys_p;
    P.has_bias = has_bias;
    P.act = act;
    // Planes smaller than half a tile are packed several to a tile: whole images for 2-D problems, consecutive depth
    // slices of one image (a divisor of the depth, so that no tile straddles two images) for 3-D problems.
    P.ipt = 1;
    if (!z_is_batch && 2 * P.Pw <= kTileM) {
        const int cap = kTileM / P.Pw;
        if (g.OD == 1) {
            P.ipt = std::min(cap, P.units); // no more images per tile than there are
        } else {
            for (int d = std::min(cap, g.OD); d >= 1; --d)
                if (g.OD % d == 0) {
                    P.ipt = d;
                    break;
                }
        }
    }
    if (max_ipt > 0) // a caller that must keep another plan's chunk size may not afford several images per raw tile
        P.ipt = std::min(P.ipt, max_ipt);
    P.tpi = (P.Pw + kTileM - 1) / kTileM;
    P.wide = (own > kTileM) ? 1 : 0;
    P.row_tiles = (own + kTileM - 1) / kTileM;
    const int xs = ow0 * P.sw - P.pw;
    P.x0 = (xs >= 0) ? (xs / 4) * 4 : -(((-xs) + 3) / 4) * 4;
    if (P.wide) {
        // one output row per tile: the box covers 128 pixels of one row (one depth slice, one image)
        const int wneed = (kTileM - 1) * P.sw + (g.T3[2] - 1) * g.dil[2] + 1 + (xs - P.x0);
        P.RW = (wneed + 3) / 4 * 4;
        P.RN = 1;
        P.RD = (g.T3[0] - 1) * g.dil[0] + 1;
        P.RH = (g.T3[1] - 1) * g.dil[1] + 1;
    } else {
        const int wneed = (own - 1) * P.sw + (g.T3[2] - 1) * g.dil[2] + 1 + (xs - P.x0);
        P.RW = (wneed + 3) / 4 * 4;
        // rows a tile touches: maximum over the tiles of one plane (in OUTPUT rows first)
        int RHo = 1;
        for (int tq = 0; tq < P.tpi; ++tq) {
            const int q_hi = std::min((tq + 1) * kTileM, P.Pw) - 1; // (whole planes when a tile holds several)
            RHo = std::max(RHo, P.ipt > 1 ? P.ohn : q_hi / P.own - tq * kTileM / P.own + 1);
        }
        P.RN = (g.OD == 1) ? P.ipt : 1;
        P.RD = ((g.OD == 1) ? 0 : (P.ipt - 1) * P.sd) + (g.T3[0] - 1) * g.dil[0] + 1;
        P.RH = (RHo - 1) * P.sh + (g.T3[1] - 1) * g.dil[1] + 1;
    }
    const int T = g.T3[0] * g.T3[1] * g.T3[2];
    if (flat) {
        // whole, unpadded planes: BC channels x all depth slices of RN images; padding is a mask over the taps
        if (P.wide || T > 32 || g.Wst != g.W)
            return fail(ctx, PETB200_ERR_UNSUPPORTED, "flat raw tiles need rows of at most 128 pixels and at most 32 taps");
        P.x0 = 0;
        P.RW = g.W, P.RH = g.H, P.RD = g.D;
        P.RN = (g.OD == 1) ? P.ipt : 1;
    } else if (P.RW > 256 || P.RH > 256 || P.RD > 256 || P.RN > 256) {
        return fail(ctx, PETB200_ERR_UNSUPPORTED, "raw activation box %dx%dx%dx%d exceeds the TMA box limit", P.RN, P.RD, P.RH, P.RW);
    }
    const size_t budget = std::min<size_t>(ctx->smem_optin, 227 * 1024) - 1024; // alignment slack
    const int forced_bc = force_bc > 0 ? force_bc : env_int("PETB200_TC_BC", 0);
    // Channels per chunk (32, or more for filters with few taps so that one raw tile still feeds several K stages) and
    // ring depths for a given tile width; false if not even one channel's raw tile fits.
    auto fit = [&](int BN) -> bool {
        P.BN = BN;
        int bc_cap = 32 * std::max(1, std::min(4, 4 / T));
        int BC = std::min(cpg, bc_cap);
        if (BC > 32)
            BC = BC / 32 * 32;
        if (forced_bc > 0)
            BC = std::min(forced_bc, cpg);
        for (;; BC = std::max(1, BC / 2)) {
            P.BC = BC;
            P.spc = (T * BC + P.ke - 1) / P.ke;
            P.nchunks = (cpg + BC - 1) / BC;
            size_t raw = (size_t)P.RN * BC * P.RD * P.RH * P.RW * 4;
            P.raw_bytes = (int)((raw + 127) / 128 * 128);
            P.NB = 2;
            P.NR = 2;
            P.a_kmajor = 0;
            P.m_rows = 0;
            bool shape_ok = true;
            if (flat) {
                // The BC*D*H*W floats of a chunk are one contiguous run: fetch it as a 2-D box [rows][w] with w a multiple
                // of 4 (16-byte rule), both extents within the TMA box limit; chunks must start on a box boundary.
                const long long L = (long long)BC * g.D * g.H * g.W;
                P.flat_w = 0;
                for (int w = 256; w >= 4 && !P.flat_w; w -= 4)
                    if (L % w == 0 && L / w <= 256)
                        P.flat_w = w, P.flat_rows = (int)(L / w);
                shape_ok = P.flat_w != 0 && cpg % BC == 0 && P.RN <= 256;
            }
            if (shape_ok && smem_layout(P).total <= budget) {
                for (; P.NB < kMaxNB; P.NB++) { // deepen the filter ring while there is room
                    P.NB++;
                    const bool fits = smem_layout(P).total <= budget;
                    P.NB--;
                    if (!fits)
                        break;
                }
                return true;
            }
            if (BC == 1 || forced_bc > 0)
                return false;
        }
    };
    const int n_img = z_is_batch ? 1 : images;
    const int mtiles = P.wide ? n_img * g.OD * ohn * P.row_tiles : ((P.units + P.ipt - 1) / P.ipt) * P.tpi;
    const int gz = z_is_batch ? images : g.groups;
    // Tile width and K split: 128-wide tiles unless the problem has too few of them for the GPU, in which case narrower
    // tiles and/or a split of K spread the same MMA work over more SMs (see est_cycles).
    const int bn_max = Fg <= 32 ? 32 : (Fg <= 64 ? 64 : 128);
    const int forced_bn = force_bn > 0 ? force_bn : env_int("PETB200_TC_BN", 0);
    if (forced_bn != 0 && forced_bn != 32 && forced_bn != 64 && forced_bn != 128)
        return fail(ctx, PETB200_ERR_INVALID, "PETB200_TC_BN must be 32, 64 or 128");
    const int want_ks = force_ksplit > 0 ? force_ksplit : env_int("PETB200_TC_KSPLIT", 0);
    double best_cycles = 0;
    IgemmParams bestP{};
    bool have = false;
    for (int bn = 128; bn >= 32; bn /= 2) {
        if (forced_bn ? bn != forced_bn : bn > bn_max)
            continue;
        P.ksplit = 1;
        if (!fit(bn))
            continue;
        const long long ctas = (long long)mtiles * ((Fg + bn - 1) / bn) * gz;
        double cyc;
        const int ks = choose_ksplit(ctx, ctas, P, core.math, want_ks, core.beside, &cyc);
        if (ks > 1) { // the landing area takes shared memory from the rings (or even from the chunk size): fit again
            P.ksplit = ks;
            if (!fit(bn))
                continue;
            if (P.nchunks < ks) {
                P.ksplit = 1;
                if (!fit(bn))
                    continue;
                cyc = est_cycles(ctx, ctas, P, core.math, 1, core.beside);
            }
        }
        if (!have || cyc < best_cycles * 0.97) { // prefer the wider tile unless the narrower one clearly wins
            have = true;
            best_cycles = cyc;
            bestP = P;
        }
    }
    if (!have)
        return fail(ctx, PETB200_ERR_UNSUPPORTED, "raw activation tile does not fit shared memory");
    P = bestP;
    // A group's last raw box then holds channels of the next group too.  They meet zero weights, but a row's largest value, which
    // decides how its halves are scaled, would be looked for among them.
    if (P.f16 && g.groups > 1 && cpg % P.BC != 0)
        return fail(ctx, PETB200_ERR_UNSUPPORTED, "halves need whole channel chunks per group, got %d channels in chunks of %d", cpg, P.BC);
    // eight consecutive K elements are channels of one filter tap: the cheap kind of gather
    P.cstride = (P.BC % 8 == 0 && env_int("PETB200_TC_TABLE", 0) == 0) ? P.RD * P.RH * P.RW : 0;
    choose_flush(core);
    if (flat && (long long)P.RN * P.BC * P.RD * P.RH * P.RW >= (1 << 24))
        return fail(ctx, PETB200_ERR_UNSUPPORTED, "flat raw tile too large for the offset table");
    const int BN = P.BN;
    const int ntiles = (Fg + BN - 1) / BN;
    choose_grid(ctx, core, mtiles, ntiles, gz, budget);
    core.smem = smem_layout(P).total + 1024;
    core.y_elems = (z_is_batch ? (long long)images : (long long)n_img) * g.F * g.OD * g.OH * g.OW;
    if (z_is_batch)
        core.y_elems = (long long)images * ys_n;
    core.Ktot = (long long)P.nchunks * P.spc * P.ke;
    core.xd[0] = g.Wst;
    core.xd[1] = g.H;
    core.xd[2] = g.D;
    core.xd[3] = g.C;
    core.xd[4] = g.N;
    // offset table for one chunk
    // Entries past the end of the chunk's K range (their packed weights are zero): -1 where the gather tests for it; in
    // plain table mode the pixel's own first element instead, so that the gather needs no test per element (the value only
    // ever meets a zero weight, and a NaN there would poison this pixel's sum anyway).
    std::vector<int> koff((size_t)P.spc * P.ke, (!flat && P.cstride == 0) ? 0 : -1);
    const int plane_w = P.RW, plane_h = P.RH * P.RW, plane_d = P.RD * plane_h;
    for (int tap = 0; tap < T; ++tap) {
        int t = tap / (g.T3[1] * g.T3[2]), r = (tap / g.T3[2]) % g.T3[1], s = tap % g.T3[2];
        for (int ci = 0; ci < P.BC; ++ci)
            koff[(size_t)tap * P.BC + ci] =
                (ci * plane_d + t * g.dil[0] * plane_h + r * g.dil[1] * plane_w + s * g.dil[2]) | (flat ? tap << 24 : 0);
    }
    core.offsets.swap(koff);
    return raise_smem_limit(ctx);
}

// fp16 halves or TF32?  Per K a stage of halves takes half the MMAs, half the handshakes and half the packed bytes; a launch costs
// 0.3 to 0.8 us more (the rows' range to be watched, 64 elements split before the first MMA).  Measured over the convolutions of
// ResNet-18 at batch 1, 8 and 64 and of ResNet3D-18, 13 others and 100 matmuls of 16 to 4096 rows, as time of fp16 over time of
// TF32, against K stages (of 32) x filters of a tile:
//   convolutions, whose gather is the slower part: 1.00 to 1.17 up to 1600 (1x1, stems, K splits at batch 1; 64 filters and 64
//   channels 1.01), 0.95 at 1800, 0.88 at 2300, 0.65 to 0.8 from 4000 on (512 channels dilated: 74 -> 48 us);
//   row-major products, times the tiles that a CTA takes in turn: 1.04 to 1.2 below 256, 0.8 to 1.1 at 256, 0.97 at 400 to 1000,
//   0.9 at 2000, 0.7 at 8000 (4096 x 4096 x 512: 70 -> 50 us).
//   A stage of halves lasts about 1.6 times one of TF32, so none of this holds where K is mostly padding: 7 channels of 1x1 to a
// chunk are one stage either way (46 us against 74), 72 values three stages or two (480 channels in chunks of 8, 36 us against 43).
// And with one stage to a chunk a transform set waits for a raw tile of its own every time (144 channels in chunks of 4, 143 us
// against 166).
//   The B of a batched product is packed in every call as a rule (a weight has no batch), which for B[b][k][n] takes 1 to 4 us more
// than for TF32: 37 x 423 x 608 x 76 (2432) 19.5 us against 21.5, 2 x 82 x 556 x 3052 (1152) 19 against 25; 4 x 500 x 770 x 1001 (3200)
// 34.1 against 31.5.  `tf32`: the plan's parameters for TF32.
static bool f16_pays(const petb200_ctx *ctx, const IgemmParams &tf32, const dim3 &grid, int batch) {
    const long long ctas = (long long)grid.x * grid.y * grid.z;
    const long long turns = tf32.pp ? (tf32.tiles + ctas - 1) / ctas : (ctas + ctx->sm_count - 1) / ctx->sm_count;
    const long long tile = (long long)((tf32.nchunks + tf32.ksplit - 1) / tf32.ksplit) * tf32.spc * tf32.BN;
    return tf32.a_kmajor ? turns * tile >= (batch > 1 ? 3000 : 300) : tile >= 1600;
}
static bool f16_fits(const IgemmParams &tf32, const IgemmParams &f16) {
    return (tf32.a_kmajor || f16.spc > 1) && 5ll * f16.nchunks * f16.spc <= 3ll * tf32.nchunks * tf32.spc;
}
// Runs `configure` for the arithmetic that the caller asks for; kMathAuto: for TF32, and again for fp16 where that pays.  What fp16
// cannot serve stays with TF32.
template <typename F> static int configure_for(petb200_ctx *ctx, TcCore &core, int math, F &&configure, int batch = 1) {
    core.math = math == kMathAuto ? kMathTf32x3 : math;
    int rc = configure();
    if (rc == PETB200_OK && math == kMathAuto && f16_pays(ctx, core.P, core.grid, batch)) {
        const IgemmParams tf32 = core.P;
        core.math = kMathF16x3;
        core.P = IgemmParams{};
        rc = configure();
        if (rc == PETB200_OK && !f16_fits(tf32, core.P))
            rc = PETB200_ERR_UNSUPPORTED;
    }
    if (rc == PETB200_ERR_UNSUPPORTED && core.math == kMathF16x3) {
        core.math = kMathTf32x3;
        core.P = IgemmParams{};
        rc = configure();
    }
    return rc;
}

// ---- exported to conv.cu -------------------------------------------------------------------------------------
struct TcConv {
    TcCore full;                 // the whole output
    ConvGeom g{};
    int has_bias = 0, act = 0;
    long long ys[3] = {0, 0, 0}; // output strides {image, filter, pixel}: {F*plane, plane, 1} (NCHW) or {F*plane, 1, F} (channels last)
    std::map<std::array<int, 4>, TcCore *> windows; // correction windows, keyed by (oh0,ohn,ow0,own)
    ~TcConv() {
        for (auto &kv : windows)
            delete kv.second;
    }
};

int tc_conv_create(petb200_ctx *ctx, int nsp, const int *in_dims, int f, const int *k, const int *pad, const int *stride,
                   const int *dil, int groups, int has_bias, int act, int passes, void **out, size_t *dev_bytes, int channels_last_out) {
    if (ctx->cc_major != 10)
        return fail(ctx, PETB200_ERR_UNSUPPORTED, "tcgen05 kernels need compute capability 10.x, device has %d.%d", ctx->cc_major, ctx->cc_minor);
    auto *t = new TcConv();
    ConvGeom &g = t->g;
    g.N = in_dims[0];
    g.C = in_dims[1];
    if (nsp == 3) {
        g.D = in_dims[2];
        g.H = in_dims[3];
        g.W = in_dims[4];
        for (int i = 0; i < 3; ++i) {
            g.T3[i] = k[i];
            g.pad[i] = pad[i];
            g.stride[i] = stride[i];
            g.dil[i] = dil[i];
        }
    } else {
        g.D = 1;
        g.H = in_dims[2];
        g.W = in_dims[3];
        g.T3[0] = 1;
        g.pad[0] = 0;
        g.stride[0] = 1;
        g.dil[0] = 1;
        for (int i = 0; i < 2; ++i) {
            g.T3[i + 1] = k[i];
            g.pad[i + 1] = pad[i];
            g.stride[i + 1] = stride[i];
            g.dil[i + 1] = dil[i];
        }
    }
    g.F = f;
    g.groups = groups;
    auto oext = [](int in, int kk, int p, int s, int d) { return (in - (kk - s) * d + 2 * p) / s; };
    g.OD = nsp == 3 ? oext(g.D, g.T3[0], g.pad[0], g.stride[0], g.dil[0]) : 1;
    g.OH = oext(g.H, g.T3[1], g.pad[1], g.stride[1], g.dil[1]);
    g.OW = oext(g.W, g.T3[2], g.pad[2], g.stride[2], g.dil[2]);
    g.Wst = g.W;
    t->has_bias = has_bias;
    t->act = act;
    t->full.ctx = ctx;
    const long long plane = (long long)g.OD * g.OH * g.OW;
    t->ys[0] = (long long)g.F * plane;
    t->ys[1] = channels_last_out ? 1 : plane;
    t->ys[2] = channels_last_out ? g.F : 1;
    // Rows that are not multiples of 16 bytes cannot be a TMA stride: small planes are fetched whole ("flat"), anything
    // else is re-pitched by the caller first (tc_conv_row_pitch tells it to what).
    int rc = configure_for(ctx, t->full, passes, [&]() {
        g.Wst = g.W;
        if (g.W % 4 != 0) {
            const int flat = tc_configure(ctx, t->full, g, 0, g.OH, 0, g.OW, 0, g.N, t->ys[0], t->ys[1], t->ys[2], has_bias, act, 0, 0, 0, 1);
            if (flat != PETB200_ERR_UNSUPPORTED)
                return flat;
            g.Wst = (g.W + 3) / 4 * 4;
            t->full.P = IgemmParams{};
        }
        return tc_configure(ctx, t->full, g, 0, g.OH, 0, g.OW, 0, g.N, t->ys[0], t->ys[1], t->ys[2], has_bias, act);
    });
    if (rc) {
        delete t;
        return rc;
    }
    TcCore &c = t->full;
    c.rows_b = g.F;
    rc = c.alloc_b();
    if (rc) {
        delete t;
        return rc;
    }
    *dev_bytes = c.whi.bytes + c.wlo.bytes + c.fscale_buf.bytes + c.koff.bytes;
    *out = t;
    return PETB200_OK;
}

// A stride-1, dilation-1 2-D convolution whose geometry is given explicitly instead of derived: signed padding (a negative
// value crops; whatever falls outside the input reads as zero on every side, so bottom/right padding is whatever the
// output extent asks for), an output window of ohn x own pixels, and free output strides {image, filter, row, pixel}
// with row = ow_nominal * pixel.  Used by the transposed convolution, whose sh*sw phases are such convolutions writing
// every sh-th row and sw-th column of a channels-last tensor.
int tc_conv_create_view(petb200_ctx *ctx, int n, int c, int h, int w, int f, int r, int s, int pad_h, int pad_w, int ohn, int own,
                        int ow_nominal, long long ys_n, long long ys_f, long long ys_p, int has_bias, int act, int passes, int beside, void **out,
                        size_t *dev_bytes) {
    if (ctx->cc_major != 10)
        return fail(ctx, PETB200_ERR_UNSUPPORTED, "tcgen05 kernels need compute capability 10.x, device has %d.%d", ctx->cc_major, ctx->cc_minor);
    if (ohn <= 0 || own <= 0 || own > ow_nominal)
        return fail(ctx, PETB200_ERR_INVALID, "conv view: empty or oversized window");
    auto *t = new TcConv();
    ConvGeom &g = t->g;
    g.N = n, g.C = c, g.D = 1, g.H = h, g.W = w, g.Wst = w, g.F = f, g.groups = 1;
    g.T3[0] = 1, g.T3[1] = r, g.T3[2] = s;
    g.pad[0] = 0, g.pad[1] = pad_h, g.pad[2] = pad_w;
    for (int i = 0; i < 3; ++i)
        g.stride[i] = 1, g.dil[i] = 1;
    g.OD = 1, g.OH = ohn, g.OW = ow_nominal;
    t->has_bias = has_bias;
    t->act = act;
    t->full.ctx = ctx;
    t->full.beside = beside;
    t->ys[0] = ys_n, t->ys[1] = ys_f, t->ys[2] = ys_p;
    int rc = configure_for(ctx, t->full, passes, [&]() {
        return tc_configure(ctx, t->full, g, 0, ohn, 0, own, 0, n, ys_n, ys_f, ys_p, has_bias, act, 0, 0, 0, w % 4 != 0);
    });
    if (rc) {
        delete t;
        return rc;
    }
    TcCore &core = t->full;
    core.rows_b = f;
    rc = core.alloc_b();
    if (rc) {
        delete t;
        return rc;
    }
    *dev_bytes = core.whi.bytes + core.wlo.bytes + core.fscale_buf.bytes + core.koff.bytes;
    *out = t;
    return PETB200_OK;
}

void tc_conv_destroy(void *h) { delete (TcConv *)h; }

int tc_conv_set_weights(void *h, const float *w, cudaStream_t s) {
    auto *t = (TcConv *)h;
    TcCore &c = t->full;
    const int cpg = t->g.C / t->g.groups, T = t->g.T3[0] * t->g.T3[1] * t->g.T3[2];
    if (c.math == kMathF16x3) {
        PackFilters g{};
        g.w = w, g.hi = c.whi.p, g.lo = c.wlo.p, g.unscale = (float *)c.fscale_buf.p, g.numbers = (uint16_t *)c.factor_word(), g.number = ++c.packings;
        g.cpg = cpg, g.T = T, g.BC = c.P.BC, g.Ktot = (int)c.Ktot;
        g.by_kc_pad.set(c.P.spc * c.P.ke), g.by_bc.set(c.P.BC);
        const int parts = std::max(1, std::min({8, 2 * c.ctx->sm_count / t->g.F, (int)((c.Ktot + 1023) / 1024)}));
        k_pack_conv_f16<<<dim3((unsigned)t->g.F, (unsigned)parts), 256, 0, s>>>(g);
        c.weights_ready = true;
        return launched(c.ctx, "k_pack_conv_f16");
    }
    long long total = (long long)t->g.F * c.Ktot;
    int blocks = (int)std::min<long long>((total + 255) / 256, (long long)c.ctx->sm_count * 16);
    auto kern = c.math == kMathBf16x3 ? k_pack_conv_w<kMathBf16x3> : (c.math == kMathTf32x1 ? k_pack_conv_w<kMathTf32x1> : k_pack_conv_w<kMathTf32x3>);
    kern<<<blocks, 256, 0, s>>>(w, c.whi.p, c.wlo.p, t->g.F, cpg, T, c.P.BC, c.P.spc * c.P.ke, c.P.nchunks);
    c.weights_ready = true;
    return launched(c.ctx, "k_pack_conv_w");
}

// One of several convolutions of the same x that fill disjoint parts of one tensor; link: its place in their chain of launches
// (0: none), where tc_conv_can_link() holds for all of them.
bool tc_conv_can_link(void *h) { return !((TcConv *)h)->full.P.pp; } // (persistent tiles fill the GPU by themselves)
int tc_conv_run_part(void *h, const float *x, const float *bias, float *y, int link, cudaStream_t s) {
    auto *t = (TcConv *)h;
    if (!t->full.weights_ready)
        return fail(t->full.ctx, PETB200_ERR_INVALID, "conv run before set_weights");
    return t->full.launch(x, bias, nullptr, y, s, link);
}

int tc_conv_run(void *h, const float *x, const float *bias, const float *res, float *y, const int *win, cudaStream_t s) {
    auto *t = (TcConv *)h;
    if (!t->full.weights_ready)
        return fail(t->full.ctx, PETB200_ERR_INVALID, "conv run before set_weights");
    if (!win)
        return t->full.launch(x, bias, res, y, s);
    const ConvGeom &g = t->g;
    if (win[0] < 0 || win[1] <= 0 || win[0] + win[1] > g.OH || win[2] < 0 || win[3] <= 0 || win[2] + win[3] > g.OW)
        return fail(t->full.ctx, PETB200_ERR_INVALID, "correction window outside the output");
    const std::array<int, 4> key = {win[0], win[1], win[2], win[3]};
    TcCore *&wc = t->windows[key];
    if (!wc) {
        wc = new TcCore();
        wc->ctx = t->full.ctx;
        wc->math = t->full.math;
        wc->packed_by = &t->full;
        // A window must consume K in exactly the order of the full operator (same BC / chunking), otherwise the
        // two would round differently; the raw box only shrinks for a window, so the full plan's BC always fits.
        int rc = tc_configure(wc->ctx, *wc, g, win[0], win[1], win[2], win[3], 0, g.N, t->ys[0], t->ys[1], t->ys[2],
                              t->has_bias, t->act, t->full.P.BC, t->full.P.ksplit, t->full.P.BN, t->full.P.flat);
        if (rc == PETB200_ERR_UNSUPPORTED) {
            // A small window packs several images into one tile, and with the full plan's chunk size forced the raw tile
            // of that many images may not fit: one image per tile always does (it is the full plan's raw tile or less).
            memset(&wc->P, 0, sizeof wc->P);
            rc = tc_configure(wc->ctx, *wc, g, win[0], win[1], win[2], win[3], 0, g.N, t->ys[0], t->ys[1], t->ys[2], t->has_bias,
                              t->act, t->full.P.BC, t->full.P.ksplit, t->full.P.BN, t->full.P.flat, std::max(1, t->full.P.ipt));
        }
        if (rc == PETB200_OK && (wc->P.BN != t->full.P.BN || wc->P.BC != t->full.P.BC || wc->Ktot != t->full.Ktot || wc->P.ksplit != t->full.P.ksplit))
            rc = fail(wc->ctx, PETB200_ERR_UNSUPPORTED, "window plan diverged from the full plan");
        if (rc == PETB200_OK)
            rc = wc->upload_offsets();
        if (rc) {
            delete wc;
            t->windows.erase(key);
            return rc;
        }
        wc->map_bhi = t->full.map_bhi;
        wc->map_blo = t->full.map_blo;
        wc->weights_ready = true;
    }
    return wc->launch(x, bias, res, y, s);
}

void tc_conv_out_dims(void *h, int *d5) {
    auto *t = (TcConv *)h;
    d5[0] = t->g.N;
    d5[1] = t->g.F;
    d5[2] = t->g.OD;
    d5[3] = t->g.OH;
    d5[4] = t->g.OW;
}
void tc_conv_set_starve(void *h, int on) { ((TcConv *)h)->full.starve = on; }
int tc_set_wait_limit_ns(unsigned long long ns) {
    for (SetWaitLimitFn set : {igemm_tf32_wait_limit, igemm_f16_wait_limit, igemm_opt_wait_limit, igemm_band_wait_limit})
        if (int rc = set(ns))
            return rc;
    return PETB200_OK;
}
int tc_conv_row_pitch(void *h) { return ((TcConv *)h)->g.Wst; }
// (halves carry TF32's significand within their range, see row_exponent: the family keeps its name)
static const char *tc_variant_name(int math) {
    return math == kMathTf32x1 ? "tc_1xtf32_ts" : (math == kMathBf16x3 ? "tc_bf16x3_ts" : (math == kMathF16x3 ? "tc_3xtf32_f16_ts" : "tc_3xtf32_ts"));
}
const char *tc_conv_variant(void *h) {
    const TcCore &c = ((TcConv *)h)->full;
    return tc_variant_name(c.math);
}

// ---- matmul on the same kernel ------------------------------------------------------------------------------
// C[b,m,n] = A·B with A supplied as [b,k,m] (i.e. transA): a 1x1 "convolution" whose image is one batch entry,
// channels = k, width = m; B is packed per call (or once, for weights) into hi/lo [b*n][Kpad].
struct TcMatmul {
    // element strides {A batch, A row, B batch, B row (of the stored matrix), C batch, C row}; innermost dims contiguous
    long long st[6] = {0, 0, 0, 0, 0, 0};
    TcCore core;
    int bs, m, n, k, transB;
    // A as passed is rows of `a_w` values that TMA cannot address: copied to a pitch of `a_pitch` first (0 rows: consumed as it is)
    long long a_rows = 0;
    int a_w = 0, a_pitch = 0;
};

// Row-major A ([b][m][k], k % 4 == 0): the kernel's K-major mode, no re-layout of A.
static int tc_configure_kmajor(petb200_ctx *ctx, TcCore &core, int bs, int m, int n, int k, int has_bias, int act,
                               const long long *st) {
    IgemmParams &P = core.P;
    memset(&P, 0, sizeof P);
    P.a_kmajor = 1;
    P.ke = core.half() ? 64 : kStageK;
    P.f16 = core.math == kMathF16x3;
    P.m_rows = m;
    P.z_is_batch = 1;
    P.OD = P.OH = 1, P.OW = m, P.ohn = 1, P.own = m, P.Pw = m, P.units = 1, P.ipt = 1, P.tpi = (m + kTileM - 1) / kTileM;
    P.sd = P.sh = P.sw = 1;
    P.cpg = k, P.Fg = n;
    P.BC = P.ke, P.spc = 1, P.nchunks = (k + P.ke - 1) / P.ke;
    P.RN = P.RD = 1, P.RH = kTileM, P.RW = kStageK;
    P.raw_bytes = kAHalfBytes * (P.ke / kStageK); // one [128][32] fp32 tile per 32 K elements of a stage
    P.ys_n = st[4], P.ys_f = 1, P.ys_p = st[5];
    core.a_batch = st[0], core.a_row = st[1];
    P.has_bias = has_bias, P.act = act;
    const size_t budget = std::min<size_t>(ctx->smem_optin, 227 * 1024) - 1024;
    P.NB = 2, P.NR = 2;
    // tile width and K split by the cycle model (before the rings are sized: a split takes shared memory)
    {
        const int bn_max = n <= 32 ? 32 : (n <= 64 ? 64 : 128), forced_bn = env_int("PETB200_TC_BN", 0);
        double best = 0;
        int best_bn = 0, best_ks = 1;
        for (int bn = 128; bn >= 32; bn /= 2) {
            if (forced_bn ? bn != forced_bn : bn > bn_max)
                continue;
            P.BN = bn;
            double cyc;
            const int ks = choose_ksplit(ctx, (long long)P.tpi * ((n + bn - 1) / bn) * bs, P, core.math,
                                         env_int("PETB200_TC_KSPLIT", 0), 1, &cyc);
            if (!best_bn || cyc < best * 0.97)
                best = cyc, best_bn = bn, best_ks = ks;
        }
        if (!best_bn)
            return fail(ctx, PETB200_ERR_INVALID, "PETB200_TC_BN must be 32, 64 or 128");
        P.BN = best_bn;
        P.ksplit = best_ks;
    }
    if (smem_layout(P).total > budget)
        return fail(ctx, PETB200_ERR_UNSUPPORTED, "matmul tile does not fit shared memory");
    for (bool grew = true; grew;) { // deepen both rings alternately: every K stage needs one B tile and one raw tile
        grew = false;
        if (P.NB < kMaxNB) {
            P.NB++;
            if (smem_layout(P).total <= budget)
                grew = true;
            else
                P.NB--;
        }
        if (P.NR < kMaxNR) {
            P.NR++;
            if (smem_layout(P).total <= budget)
                grew = true;
            else
                P.NR--;
        }
    }
    choose_flush(core);
    choose_grid(ctx, core, P.tpi, (n + P.BN - 1) / P.BN, bs, budget);
    core.smem = smem_layout(P).total + 1024;
    core.Ktot = (long long)P.nchunks * P.ke;
    core.xd[0] = k, core.xd[1] = m, core.xd[2] = bs;
    std::vector<int> koff(P.ke, -1); // unused in this mode; the kernel still copies one stage worth of table
    core.offsets.swap(koff);
    core.y_elems = (long long)bs * m * n;
    return raise_smem_limit(ctx);
}

int tc_matmul_create(petb200_ctx *ctx, int bs, int m, int n, int k, int transA, int transB, int has_bias, int act, int passes,
                     const long long *strides, void **out, size_t *dev_bytes) {
    const int mp = (m + 3) / 4 * 4; // row pitch of A as [b][k][mp]
    if (ctx->cc_major != 10)
        return fail(ctx, PETB200_ERR_UNSUPPORTED, "tcgen05 kernels need compute capability 10.x");
    auto *t = new TcMatmul();
    t->bs = bs;
    t->m = m;
    t->n = n;
    t->k = k;
    t->transB = transB;
    t->core.ctx = ctx;
    const long long dense[6] = {(long long)m * k, transA ? m : k, (long long)k * n, transB ? k : n, (long long)m * n, n};
    for (int i = 0; i < 6; ++i)
        t->st[i] = strides ? strides[i] : dense[i];
    int rc;
    if (!transA && k % 4 == 0 && t->st[0] % 4 == 0 && t->st[1] % 4 == 0) {
        rc = configure_for(ctx, t->core, passes, [&]() { return tc_configure_kmajor(ctx, t->core, bs, m, n, k, has_bias, act, t->st); }, bs);
    } else if (!transA && !strides) { // rows of A off the 16-byte grid: the same on a copy with a pitch of whole 16-byte pieces
        t->a_rows = (long long)bs * m, t->a_w = k, t->a_pitch = (k + 3) / 4 * 4;
        const long long st[6] = {(long long)m * t->a_pitch, t->a_pitch, t->st[2], t->st[3], t->st[4], t->st[5]};
        rc = configure_for(ctx, t->core, passes, [&]() { return tc_configure_kmajor(ctx, t->core, bs, m, n, t->a_pitch, has_bias, act, st); }, bs);
    } else if (strides) {
        delete t;
        return fail(ctx, PETB200_ERR_UNSUPPORTED, "strided matmul operands need row-major A with k and the A strides multiples of 4");
    } else {
        if (m % 4 != 0)
            t->a_rows = (long long)bs * k, t->a_w = m, t->a_pitch = mp;
        ConvGeom g{};
        g.N = bs;
        g.C = k;
        g.D = 1;
        g.H = 1;
        g.W = m;
        g.Wst = mp;
        g.F = n;
        g.groups = 1;
        for (int i = 0; i < 3; ++i) {
            g.T3[i] = 1;
            g.pad[i] = 0;
            g.stride[i] = 1;
            g.dil[i] = 1;
        }
        g.OD = 1;
        g.OH = 1;
        g.OW = m;
        rc = configure_for(ctx, t->core, passes, [&]() { return tc_configure(ctx, t->core, g, 0, 1, 0, m, 1, bs, (long long)m * n, 1, n, has_bias, act); });
    }
    if (rc) {
        delete t;
        return rc;
    }
    TcCore &c = t->core;
    c.rows_b = bs * n;
    // rows of different batch entries are adjacent: Fg = n rows per z
    rc = c.alloc_b();
    if (rc) {
        delete t;
        return rc;
    }
    *dev_bytes = c.whi.bytes + c.wlo.bytes + c.fscale_buf.bytes + c.koff.bytes;
    *out = t;
    return PETB200_OK;
}
// G2BMM on the tensor-core kernel (dilation 1): q [bs][n][m] is the row-major A operand, the keys k [bs][n][m] are packed like
// a matmul's B operand ([bs*n rows][K]); a CTA column (blockIdx.y) is one 64-key piece of the 2w + 128 keys a row tile can
// meet, and CTAs walk the row tiles in persistent mode.  `y` [bs][n][2w+1] is written by the banded epilogue.
int tc_g2bmm_create(petb200_ctx *ctx, int bs, int n, int m, int w, void **out) {
    if (ctx->cc_major != 10)
        return fail(ctx, PETB200_ERR_UNSUPPORTED, "tcgen05 kernels need compute capability 10.x");
    if (m % 4 != 0 || w <= 0)
        return fail(ctx, PETB200_ERR_UNSUPPORTED, "tensor-core g2bmm needs m divisible by 4");
    auto *t = new TcMatmul();
    t->bs = bs, t->m = n, t->n = n, t->k = m, t->transB = 1;
    t->st[2] = (long long)n * m, t->st[3] = m; // keys: batch and row strides
    TcCore &core = t->core;
    core.ctx = ctx;
    IgemmParams &P = core.P;
    memset(&P, 0, sizeof P);
    P.a_kmajor = 1, P.ke = kStageK, P.m_rows = n, P.z_is_batch = 1, P.band_w = w, P.band_g2 = 1;
    P.OD = P.OH = 1, P.OW = n, P.ohn = 1, P.own = n, P.Pw = n, P.units = 1, P.ipt = 1, P.tpi = (n + kTileM - 1) / kTileM;
    P.sd = P.sh = P.sw = 1;
    P.cpg = m, P.Fg = n, P.BN = 64, P.ksplit = 1;
    P.BC = P.ke, P.spc = 1, P.nchunks = (m + P.ke - 1) / P.ke;
    P.RN = P.RD = 1, P.RH = kTileM, P.RW = kStageK, P.raw_bytes = kAHalfBytes;
    P.ys_n = (long long)n * (2 * w + 1), P.ys_f = 1, P.ys_p = 2 * w + 1;
    core.a_batch = (long long)n * m, core.a_row = m;
    P.fl = 0;
    const int key_tiles = (2 * w + kTileM + P.BN - 1) / P.BN;
    P.pp = 1, P.ntiles = key_tiles, P.mtiles = P.tpi, P.tiles = P.tpi * key_tiles * bs;
    const size_t budget = std::min<size_t>(ctx->smem_optin, 227 * 1024) - 1024;
    P.NB = 2, P.NR = 2;
    if (smem_layout(P).total > budget) {
        delete t;
        return fail(ctx, PETB200_ERR_UNSUPPORTED, "g2bmm tile does not fit shared memory");
    }
    for (bool grew = true; grew;) {
        grew = false;
        if (P.NB < kMaxNB) {
            P.NB++;
            if (smem_layout(P).total <= budget)
                grew = true;
            else
                P.NB--;
        }
        if (P.NR < kMaxNR) {
            P.NR++;
            if (smem_layout(P).total <= budget)
                grew = true;
            else
                P.NR--;
        }
    }
    core.smem = smem_layout(P).total + 1024;
    core.Ktot = (long long)P.nchunks * P.ke;
    core.xd[0] = m, core.xd[1] = n, core.xd[2] = bs;
    core.offsets.assign(P.ke, -1);
    core.grid = dim3((unsigned)std::min(P.tiles, ctx->sm_count), 1u, 1u);
    core.y_elems = (long long)bs * n * (2 * w + 1);
    core.rows_b = bs * n;
    int rc = raise_smem_limit(ctx);
    if (rc == PETB200_OK)
        rc = core.alloc_b();
    if (rc) {
        delete t;
        return rc;
    }
    if (env_int("PETB200_TC_VERBOSE", 0))
        fprintf(stderr, "[petb200] g2bmm plan: grid %u x %u x %u, NB %d NR %d\n", core.grid.x, core.grid.y, core.grid.z, P.NB, P.NR);
    *out = t;
    return PETB200_OK;
}

// GBMML on the tensor-core kernel (dilation 1): y [bs][n][m] = band p [bs][n][2w+1] times the value rows v [bs][n][m] it points at.
// Rows are the M dimension, v's columns the filters (packed like a matmul's B operand with the keys as K), and the K range
// of a row tile is the key window [128*tile - w, 128*tile + 127 + w]; the transform threads read the band from global memory.
int tc_gbmml_create(petb200_ctx *ctx, int bs, int n, int m, int w, void **out) {
    if (ctx->cc_major != 10)
        return fail(ctx, PETB200_ERR_UNSUPPORTED, "tcgen05 kernels need compute capability 10.x");
    if (m % 4 != 0 || m > 128 || w < 3) // (w: see band_copy)
        return fail(ctx, PETB200_ERR_UNSUPPORTED, "tensor-core gbmml needs m divisible by 4 and at most 128, and a width of 3 or more");
    auto *t = new TcMatmul();
    t->bs = bs, t->m = n, t->n = m, t->k = n, t->transB = 0;
    t->st[2] = (long long)n * m, t->st[3] = m; // v: batch stride, stride of a key row
    TcCore &core = t->core;
    core.ctx = ctx;
    IgemmParams &P = core.P;
    memset(&P, 0, sizeof P);
    P.a_kmajor = 1, P.ke = kStageK, P.m_rows = n, P.z_is_batch = 1, P.band_w = w;
    P.OD = P.OH = 1, P.OW = n, P.ohn = 1, P.own = n, P.Pw = n, P.units = 1, P.ipt = 1, P.tpi = (n + kTileM - 1) / kTileM;
    P.sd = P.sh = P.sw = 1;
    P.cpg = n, P.Fg = m, P.BN = m <= 32 ? 32 : (m <= 64 ? 64 : 128), P.ksplit = 1;
    // a chunk is two K stages of a row tile's key window (whose start is rounded down to a multiple of 4)
    P.BC = kBandKeys, P.spc = kBandStages, P.nchunks = (2 * w + kTileM + 3 + kBandKeys - 1) / kBandKeys;
    P.RN = P.RD = 1, P.RH = kTileM, P.RW = kStageK, P.raw_bytes = kTileM * kBandPitch * 4;
    P.band_words = (long long)bs * n * (2 * w + 1);
    P.ys_n = (long long)n * m, P.ys_f = 1, P.ys_p = m;
    P.NB = 2, P.NR = 2;
    const size_t budget = std::min<size_t>(ctx->smem_optin, 227 * 1024) - 1024;
    if (smem_layout(P).total > budget) {
        delete t;
        return fail(ctx, PETB200_ERR_UNSUPPORTED, "gbmml tile does not fit shared memory");
    }
    for (bool grew = true; grew;) {
        grew = false;
        for (int *ring : {&P.NR, &P.NB}) {
            if (*ring >= 4)
                continue;
            ++*ring;
            if (smem_layout(P).total <= budget)
                grew = true;
            else
                --*ring;
        }
    }
    choose_flush(core);
    choose_grid(ctx, core, P.tpi, (m + P.BN - 1) / P.BN, bs, budget);
    core.smem = smem_layout(P).total + 1024;
    core.Ktot = ((long long)n + P.ke - 1) / P.ke * P.ke; // the packed operand covers all keys; a tile reads its window of them
    core.xd[0] = kStageK, core.xd[1] = kTileM, core.xd[2] = 1; // (the activation map is not used: any valid extents)
    core.a_batch = kStageK * kTileM, core.a_row = kStageK;
    core.offsets.assign(P.spc * P.ke, -1);
    core.y_elems = (long long)bs * n * m;
    core.rows_b = bs * m;
    int rc = raise_smem_limit(ctx);
    if (rc == PETB200_OK)
        rc = core.alloc_b();
    if (rc) {
        delete t;
        return rc;
    }
    *out = t;
    return PETB200_OK;
}
// runs a GBMML plan: `p` is the band, `y` the result (the values v were packed by tc_matmul_pack_b)
int tc_gbmml_run(void *h, const float *p, float *y, cudaStream_t s) {
    auto *t = (TcMatmul *)h;
    t->core.P.band_p = p;
    return t->core.launch(p, nullptr, nullptr, y, s); // (the activation map is encoded over p but never used by this mode)
}

// Words of the copy of A that a call needs (0: A is consumed as it is).
long long tc_matmul_a_copy(void *h) {
    auto *t = (TcMatmul *)h;
    return t->a_rows * t->a_pitch;
}
const char *tc_matmul_variant(void *h) { return tc_variant_name(((TcMatmul *)h)->core.math); }
void tc_matmul_destroy(void *h) { delete (TcMatmul *)h; }
// Packs B (null: it has been) and copies A to an addressable pitch (null: not needed), in one launch.
int tc_matmul_prepare(void *h, const float *b, const float *a, float *a_copy, cudaStream_t s) {
    auto *t = (TcMatmul *)h;
    TcCore &c = t->core;
    const bool f16 = c.math == kMathF16x3;
    PrepareArgs g{};
    g.b = b, g.hi = c.whi.p, g.lo = c.wlo.p, g.bs = t->bs, g.n = t->n, g.k = t->k, g.Kpad = (int)c.Ktot;
    if (f16)
        g.unscale = (float *)c.fscale_buf.p, g.numbers = (uint16_t *)c.factor_word(), g.number = b ? ++c.packings : (uint16_t)0;
    g.BC = c.P.BC, g.sb_batch = t->st[2], g.sb_row = t->st[3];
    g.tiles_k = g.Kpad / (f16 ? kPrepUnit : 32); // (Kpad is a multiple of the stage's K)
    const int width = f16 && (t->n + 31) / 32 * (long long)t->bs * std::min(8, g.tiles_k) < 2ll * c.ctx->sm_count ? 8 : 32; // of a strip of columns
    g.tiles_n = (t->n + width - 1) / width;
    g.by_kc_pad.set(c.P.spc * c.P.ke), g.by_tiles_k.set(g.tiles_k), g.by_tiles_n.set(g.tiles_n);
    g.split = 1;
    const long long strips = (long long)g.tiles_n * t->bs, rows = (long long)t->n * t->bs;
    long long tiles = (long long)g.tiles_k * strips;
    if (f16 && t->transB) { // a row's units stay in registers, and there are sixteen warps for every SM
        while (g.split < 8 && 2 * g.split <= g.tiles_k && (g.tiles_k > g.split * kPrepKeep || rows * g.split < 16ll * c.ctx->sm_count))
            g.split *= 2;
        tiles = (rows * g.split + 7) / 8;
    } else if (f16) { // a strip's units stay in shared memory, and there are two CTAs for every SM
        while (g.split < 8 && 2 * g.split <= g.tiles_k && (g.tiles_k > g.split * kPrepKeep || strips * g.split < 2ll * c.ctx->sm_count))
            g.split *= 2;
        tiles = strips * g.split;
    }
    if (!b)
        tiles = 0;
    if (tiles > (1 << 30))
        return fail(c.ctx, PETB200_ERR_UNSUPPORTED, "matmul operand too large to pack in one launch");
    g.b_tiles = (int)tiles;
    g.a = a, g.a_copy = a_copy, g.a_rows = a ? t->a_rows : 0, g.a_w = t->a_w, g.a_pitch = t->a_pitch;
    long long a_blocks = std::min<long long>((g.a_rows + 7) / 8, (long long)c.ctx->sm_count * 8);
    if (tiles + a_blocks == 0)
        return PETB200_OK;
    if (f16 && !t->transB) {
        a_blocks = (a_blocks + g.split - 1) / g.split * g.split; // whole clusters
        const int units = (g.tiles_k + g.split - 1) / g.split;
        const size_t smem = (size_t)(width == 32 ? std::min(kPrepRoom<32>, units) * kPrepPitch<32> : std::min(kPrepRoom<8>, units) * kPrepPitch<8>)*kPrepUnit * 4;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((unsigned)(tiles + a_blocks)), cfg.blockDim = dim3(256), cfg.dynamicSmemBytes = smem, cfg.stream = s;
        cudaLaunchAttribute attr[2] = {};
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)g.split, attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr, cfg.numAttrs = pdl_enabled() ? 2 : 1;
        (void)cudaLaunchKernelEx(&cfg, width == 32 ? k_prepare_f16_kn<32> : k_prepare_f16_kn<8>, g); // (errors surface through launched())
    } else {
        const dim3 grid((unsigned)(tiles + a_blocks));
        auto pick = [&](auto math) {
            constexpr int MATH = decltype(math)::value;
            return t->transB ? k_prepare_mm<MATH, true> : k_prepare_mm<MATH, false>;
        };
        launch_pdl(f16 ? (g.tiles_k <= g.split ? k_prepare_f16_nk<1> : k_prepare_f16_nk<kPrepKeep>) : (c.math == kMathBf16x3 ? pick(std::integral_constant<int, kMathBf16x3>())
                     : (c.math == kMathTf32x1 ? pick(std::integral_constant<int, kMathTf32x1>()) : pick(std::integral_constant<int, kMathTf32x3>()))),
                   grid, 256, 0, s, g);
    }
    if (b)
        c.weights_ready = true;
    return launched(c.ctx, f16 ? "k_prepare_f16" : "k_prepare_mm");
}
int tc_matmul_pack_b(void *h, const float *b, cudaStream_t s) { return tc_matmul_prepare(h, b, nullptr, nullptr, s); }
int tc_matmul_run(void *h, const float *a_t, const float *bias, const float *res, float *cmat, cudaStream_t s) {
    auto *t = (TcMatmul *)h;
    return t->core.launch(a_t, bias, res, cmat, s);
}

} // namespace petb200
