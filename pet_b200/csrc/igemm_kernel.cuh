// Implicit-GEMM convolution / matmul on the 5th-generation tensor cores (tcgen05) with error-compensated TF32 or fp16.
//
//   D[pixel, filter] = sum_k A[pixel, k] * B[filter, k]            k = (channel chunk, tap, channel in chunk)
//
// A tile is 128 pixels x BN filters (BN = 32, 64 or 128); a CTA computes one, or several in turn (persistent tiles).  The fp32
// accumulators and the A operand live in tensor memory (TMEM).  Sixteen warps:
//   0      TMA producer for the packed weights: per K stage (32 words of K) one 2-D tile of B_hi and one of B_lo, straight into
//          128-byte-swizzled K-major shared memory.
//   1      one thread issues, per K=8 step (K=16 of halves), the three products of 3xTF32 as two MMAs — A_hi x [B_hi;B_lo] (one MMA of width
//          2*BN: the hi*hi sum and the hi*lo sum in adjacent accumulators) and A_lo x B_hi — and commits the stage release
//          barriers.
//   2      TMA producer for the RAW activation tile of one channel chunk (all taps share it): a 5-D box
//          [images, channels, depth, rows, cols] of the NC(D)HW input, zero-filled outside the tensor, which is exactly the
//          convolution's zero padding.  Box start along W is rounded down to 16 bytes.  (3 is idle.)
//   4-7, 8-11  two transform sets taking alternate K stages.  Thread p owns pixel p of the tile: for every K stage it gathers its
//          32 values (64 for halves) from the raw tile (fixed strides where the channel chunk allows, else through a precomputed offset table:
//          tap shift, dilation, channel plane), splits each fp32 into hi (top 19 bits, or a half) and lo = x - hi, and writes both to
//          TMEM with tcgen05.st, which leaves the shared-memory read port to B alone.  With one tile per CTA they also store it.
//   12-15  drain warps.  The tensor core truncates its fp32 accumulator after every MMA, so long K ranges empty the main
//          accumulator every few stages into a running total that these warps hold.  With persistent tiles they store a finished
//          tile (tcgen05.ld -> +bias -> activation -> global stores in the way the layout of y allows, see store_block) while
//          the transform sets run on into the next.
//
// Variants (template parameters): 3xTF32 and the same three products of fp16 halves (64 K elements per stage, K = 16 per MMA;
// the host takes whichever is faster for the shape), one TF32 pass, error-compensated bf16; one tile per CTA or persistent
// tiles; the banded products.
// Split-K: the ksplit CTAs of one output tile form a thread-block cluster and exchange their partial sums through
// distributed shared memory (pushes into the owner's landing area, one cluster barrier, reduction in rank order).
// Every wait on an mbarrier is bounded (~2 s) and reports through a status word instead of hanging the GPU.
// TMA loads are per CTA (no cluster-wide loads of any kind).
#pragma once
#include "common.h"
#include "tc_ptx.cuh"
#include <cstdlib>
#include <type_traits>

namespace petb200 {

constexpr int kTileM = 128;
constexpr int kStageK = 32;               // 32-bit words per K stage = one 128-byte swizzle row (32 TF32 values or 64 halves)
// values of the kernel's PASSES parameter: error-compensated TF32 (three products per multiply), one TF32 product, and
// error-compensated bf16 (hi/lo bf16 halves, three products, K = 16 per instruction: half the MMAs of 3xTF32 per K)
// error-compensated fp16: a half holds TF32's eleven significant bits, so the same three products with K = 16 per instruction;
// what a half lacks is range, see row_exponent.
constexpr int kMathTf32x3 = 3, kMathTf32x1 = 1, kMathBf16x3 = 16, kMathF16x3 = 17;
constexpr int kMathAuto = 0; // (host side: fp16 where it is the faster one, else TF32)
constexpr int kAHalfBytes = kTileM * 128; // one 128 x 32 operand tile
// Warps: 0 filter producer, 1 MMA, 2 raw producer (3 idle); 4-7 and 8-11 the two transform sets; 12-15 the drain warps.  Each
// group of four covers the four lane quarters of TMEM.
constexpr int kThreads = 512, kSetWarp = 4, kDrainWarp = 12;
constexpr int kNA = 4; // A stages in TMEM: a transform set owns slots `set` and `set + 2`
// Kernel modes.  Single: one tile per CTA.  Persistent: a CTA walks several tiles, the transform sets run on into the next tile
// while the drain warps store the last one; with BN <= 64 and no accumulator flush (narrow) accumulators alternate between two
// TMEM regions, otherwise (wide) the drain warps take the sums of the one region into registers and hand it back first.
enum { kSingle = 0, kNarrow = 1, kWide = 2 };
// Registers per thread of the four warp groups (512 in sum, what the block is launched with): drain warps that keep a row of 128
// sums need 184 or more; in single-tile mode the transform sets also run the epilogue.
// The compiler sees one limit for all roles (128 a thread): at most 48 bytes spilled / 190 loaded; the narrow TF32 instances and the
// single-tile convolution spill nothing.
template <int PP> struct Regs {
    static constexpr int control = PP == kSingle ? 56 : 72, set = PP == kSingle ? 136 : (PP == kNarrow ? 144 : 120),
                         drain = PP == kSingle ? 184 : (PP == kNarrow ? 152 : 200);
    static_assert(control + 2 * set + drain <= 512, "more registers than the block was launched with: setmaxnreg would wait forever");
};
constexpr int kMaxNB = 6;
constexpr int kMaxNR = 6;

// Division by a number fixed when the plan is made: q = (umulhi(n, m) + n) >> s for 0 <= n < 2^31.  Tile coordinates take half a
// dozen divisions in each of four roles; as generic divisions they are more instructions per tile than a K stage, and the
// persistent kernel's roles together then overflow the SM's instruction cache.
struct FastDiv {
    uint32_t d, m, s;
    void set(int div) {
        d = (uint32_t)(div > 0 ? div : 1);
        for (s = 0; (1ull << s) < d; ++s) {
        }
        m = (uint32_t)(((1ull << 32) * ((1ull << s) - d)) / d + 1);
    }
#ifdef __CUDACC__
    __device__ __forceinline__ int div(int n) const { return (int)((__umulhi((uint32_t)n, m) + (uint32_t)n) >> s); }
#endif
};

constexpr uint32_t kBarBytes = 384;
constexpr int kExpSlots = 8;
struct SmemLayout {
    uint32_t b_off, raw_off, koff_off, split_off, stage_off, bar_off, exp_off, total;
};
// Launches in one stream that write disjoint parts of y and read only what was written before the first of them run side by side
// under programmatic dependent launch (without it they run one after the other, which gives the same).
enum { kLinkNone = 0, kLinkFirst = 1, kLinkNext = 2 };
struct IgemmParams {
    int link;               // position in such a chain
    // Made by finish_params: what a CTA would else work out, in code that every launch fetches anew and every role waits for (the
    // two 64-bit divisions of the K split and the layout of shared memory alone were 0.2 us of a launch).
    FastDiv by_tpi, by_pw, by_od, by_own;
    SmemLayout L;
    int ks_log, cols;            // ksplit = 1 << ks_log; columns of the tile that one CTA of a cluster sums
    int Pw, units;          // pixels of one output plane (one image, one depth slice); number of such planes
    int OD, OH, OW;         // full output extents (for addressing y)
    int ohn, own, oh0, ow0; // output window actually computed (ohn*own = Pw)
    int sd, sh, sw, pd, ph, pw;
    int x0;                 // box origin along W (multiple of 4, may be negative)
    int RN, RD, RH, RW, BC; // raw box extents
    int nchunks, spc;       // channel chunks; K stages per chunk
    int ke;                 // K elements per stage: 32 (TF32) or 64 (fp16 and bf16, two per 32-bit word)
    int f16;                // error-compensated fp16
    const float *fscale;    // fp16: what each packed filter has to be multiplied by (a power of two, mostly 1)
    const uint32_t *factor_word; // its halves are equal if one of them is not 1 (see TcCore::factor_word)
    int cpg, Fg, BN;        // channels per group, filters per group, tile N
    int z_is_batch;         // blockIdx.z: 0 = conv group, 1 = matmul batch
    int wide, row_tiles;    // wide mode: a tile is 128 consecutive pixels of ONE output row (rows wider than a tile)
    int tpi, ipt;           // otherwise: tiles per plane (plane larger than a tile) or whole planes per tile
    int ksplit;             // K is split over this many CTAs, launched as one thread-block cluster (2, 4, 8 or 16); partial
                            // tiles are added up through distributed shared memory
    int NB, NR;             // ring depths: B stages, raw activation buffers
    int fl;                 // 3xTF32 only: every `fl` K stages the main accumulator is drained into a running total that
                            // is summed with round-to-nearest adds (0: never).  The tensor core truncates its accumulator
                            // after every MMA; restarting it keeps the truncated partial sums short and small
    int a_kmajor;           // matmul with row-major A: the raw tile is [128 rows][32 k], 128B-swizzled, one per K stage
    int m_rows;             // a_kmajor: rows of A per batch entry
    int raw_bytes;          // bytes of one raw buffer (128-aligned)
    int flat;               // rows of the input are not 16-byte multiples: the raw tile is BC whole channels of RN images,
                            // dense and unpadded, fetched as a 2-D box [flat_rows][flat_w] of the contiguous run; padding
                            // becomes a per-pixel mask over the filter taps (<= 32 taps)
    int flat_w, flat_rows;
    int cstride;            // BC % 8 == 0: floats between consecutive channels of the raw tile (else 0: table)
    long long ys_n, ys_f, ys_p;
    int act, has_bias;
    const int *koff;
    const float *bias;
    const float *res; // optional residual, laid out like y: y = act(sum + bias + res)
    float *y;
    int *status;
    int pp;          // persistent mode: a one-dimensional grid of at most one CTA per SM walks all output tiles, CTA i tiles i,
                     // i + gridDim.x, ...
    int tiles, ntiles, mtiles; // persistent mode: all tiles, filter tiles (they vary fastest), pixel tiles
    int band_g2;     // the banded product is G2BMM (host side)
    int band_w;      // > 0: banded product y[b,i,j] = q[b,i,:] . k[b,i+j-w,:] (row-major A = q, "filters" = the keys of the window
                     // [128*tile - w, 128*tile + 127 + w] of the tile's rows, the filter tile being a 64-key piece of that window); the
                     // epilogue stores the band entries of each row at their skewed positions, zero where the key is outside [0,n)
    long long band_words; // GBMML: words of the whole band
    const float *band_p; // non-null: GBMML y[b,i,c] = sum_j p[b,i,j] * v[b,i+j-w,c]: the A operand is the band p [bs][n][2w+1] read
                     // row by row with asynchronous copies (row i of the tile meets key k through p[i][k-i+w]),
                     // the "filters" are v's columns with the keys as K (window of the tile's rows, start rounded down to 4)
    int starve;      // test hook: the filter producer announces more bytes than it loads, so the stage never completes
    // What an ordinary tile of a CTA of its own does not read.  Parameters come through the constant cache line by line, and every
    // launch waits for those it reads: with these among the others a 64-channel 3x3 layer at batch 1 took 8.44 us, now 8.36.
    FastDiv by_ntiles, by_mtiles, by_ohn, by_row_tiles, by_fl;
    int tiles_each, tiles_extra; // persistent mode: tiles of every CTA, CTAs that have one more
    int T3[3], dil[3];           // filter extents and dilations (flat only: for the tap mask)
    int xD, xH, xW;              // input extents (flat only)
};

inline SmemLayout smem_layout(const IgemmParams &P) {
    SmemLayout L;
    uint32_t o = 0;
    L.b_off = o;
    o += (uint32_t)P.NB * 2 * (uint32_t)P.BN * 128;
    L.raw_off = o;
    o += (uint32_t)P.NR * (uint32_t)P.raw_bytes;
    L.koff_off = o;
    o += (uint32_t)P.spc * (uint32_t)P.ke * 4;
    // split-K: landing area for the cluster's partial sums of this CTA's columns, [rank][BN/ksplit][128] floats.  Its
    // own region: peers push into it while this CTA may still be in its main loop.
    L.split_off = (o + 127) & ~127u;
    o = L.split_off + (P.ksplit > 1 ? 512u * (uint32_t)P.BN + 1024u : 0u); // + each tile row's offset in y (-1: none)
    // Transposition blocks of the warps that store.  Persistent mode: the drain warps' own room (the B ring is never idle).
    // Otherwise the eight transform warps use the B ring, unless it is too small (or the sums go through the cluster).
    const bool in_ring = P.ksplit > 1 || (uint32_t)P.NB * 2 * (uint32_t)P.BN * 128 >= 8u * 4096u;
    L.stage_off = (o + 127) & ~127u;
    L.bar_off = L.stage_off + (P.pp ? 4u * 4096u : (in_ring ? 0u : 8u * 4096u));
    // fp16: a second set of barriers (for the pass that repeats a tile) and the exponents of each row's largest value
    L.exp_off = L.bar_off + (P.f16 ? 2u : 1u) * kBarBytes;
    L.total = L.exp_off + (P.f16 ? (uint32_t)kExpSlots * 2u * kTileM : 0u);
    return L;
}

inline void finish_params(IgemmParams &P, unsigned grid_x) {
    P.by_ntiles.set(P.ntiles), P.by_mtiles.set(P.mtiles), P.by_tpi.set(P.tpi), P.by_pw.set(P.Pw);
    P.by_od.set(P.OD), P.by_own.set(P.own), P.by_ohn.set(P.ohn), P.by_row_tiles.set(P.row_tiles), P.by_fl.set(P.fl);
    P.L = smem_layout(P);
    for (P.ks_log = 0; (1 << P.ks_log) < P.ksplit; ++P.ks_log) {
    }
    P.cols = P.BN / P.ksplit;
    P.tiles_each = P.pp ? P.tiles / (int)grid_x : 1, P.tiles_extra = P.pp ? P.tiles % (int)grid_x : 0;
}

template <int ACT> __device__ __forceinline__ float act_fn(float v) {
    if (ACT == PETB200_ACT_RELU)
        return fmaxf(v, 0.f);
    if (ACT == PETB200_ACT_SIGMOID)
        return 1.f / (1.f + expf(-v));
    if (ACT == PETB200_ACT_TANH)
        return tanhf(v);
    if (ACT == PETB200_ACT_GELU)
        return 0.5f * v * (1.f + erff(v * 0.70710678118654752440f));
    return v;
}

// Banded product: the tile holds rows [128*bx, +128) x keys [128*bx - w + col_base, + BN) of q . k^T.  Entry (row pr, column c)
// is band column jb = col_base + c - pr of row i = 128*bx + pr (key i + jb - w); entries with jb outside [0, 2w] are not part
// of the band, entries whose key is outside [0, n) are stored as zero.  A warp passes 32 rows x 32 columns through shared
// memory (XOR-swizzled, conflict-free both ways) so that each store instruction writes 32 consecutive band columns of one row.
template <int PASSES>
__device__ __forceinline__ void epilogue_banded(uint32_t tacc, uint32_t tcross, int c_lo, int c_hi /*columns of the tile to store*/, int col_base,
                                                int p0, int bx, int zb, int n, int w, float *y, float *stage, int lane) {
    uint32_t nx[32], sm[32];
    const int bw = 2 * w + 1;
    const int i0 = bx * kTileM + p0;    // first row of this warp
    const int rows = min(32, n - i0);   // rows of it inside the tensor
    for (int cc = c_lo; cc < c_hi; cc += 32) {
        const int lo = col_base + cc - p0; // jb of (row 0, lane 0); the block spans jb in [lo - 31, lo + 31]
        if (rows <= 0 || lo + 31 < 0 || lo - 31 >= bw)
            continue; // nothing of this block lies in the band
        ptx::tmem_ld_32x32(tacc + (uint32_t)cc, nx);
        if (PASSES != kMathTf32x1)
            ptx::tmem_ld_32x32(tcross + (uint32_t)cc, sm);
        // this lane's column: band column of warp row r is jb0 - r, the key is the same for every row
        const int jb0 = col_base + cc + lane - p0, key = i0 + jb0 - w;
        const bool key_ok = key >= 0 && key < n;
        float *dst = y + ((long long)zb * n + i0) * bw + jb0; // row r: dst + r * (bw - 1)
        ptx::tmem_ld_wait();
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            const float v = PASSES != kMathTf32x1 ? __uint_as_float(nx[j]) + __uint_as_float(sm[j]) : __uint_as_float(nx[j]);
            stage[lane * 32 + (j ^ lane)] = v;
        }
        __syncwarp();
        // every entry of the block inside the band and the tensor (the common case): no tests per store
        if (rows == 32 && lo - 31 >= 0 && lo + 31 < bw && __all_sync(0xffffffffu, key_ok)) {
#pragma unroll
            for (int r = 0; r < 32; ++r, dst += bw - 1)
                *dst = stage[r * 32 + (lane ^ r)];
        } else {
#pragma unroll 4
            for (int r = 0; r < 32; ++r, dst += bw - 1)
                if (r < rows && (unsigned)(jb0 - r) < (unsigned)bw)
                    *dst = key_ok ? stage[r * 32 + (lane ^ r)] : 0.f;
        }
    }
}

// Range of the halves.  A value x is split as y = x * 2^7 (a filter's: * 2^9), hi = half(y), lo = half((y - hi) * 2^11).  hi has all of its
// eleven bits from |y| = 2^-14 on; below, hi has fewer, and what the three products leave out, lo times lo, is no longer below 2^-22
// of the product.  The units put the range of ordinary operands, [2^-21, 2^8) and [2^-23, 2^6), over that of such halves.  (Split as
// they were, rows with a 1 that meets zero weights and the rest at 1e-6 had an error of 3.3e-6, such filters 9.3e-6; now both have
// 1.5e-7 and 2 to 3e-7 with the rest at 1e-7, against 4.3e-7 with TF32.  The products with the units cost 1 to 3 % of a launch.)
// A row of A (one output pixel's operands) whose largest magnitude lies in [2^-12, 2^8) is split with the factor 1.  (The lower end
// holds the probabilities of 4096 equal keys.)  Any other row would lose digits or overflow.  So the transform threads follow the
// largest magnitude of what they split and leave its exponent beside every stage (a test for the tile's last stage would be a branch
// per stage, which costs more); whoever stores 32 rows looks at theirs first and, if one is out of range, stores nothing and asks for a second
// pass: the CTA's tiles once more with rows out of range multiplied by a power of two, which is taken out again when the sums are
// stored.  A CTA of more tiles than the exponents of kExpSlots tell has each twice in a row there, the first time for its exponents.
// Only what the first pass left is stored.  (All rows at 1e-5, ordinary rows, 3xTF32: 384 x 3072 x 768 21 / 11 / 13 us, 64 images of
// 128 x 28 x 28 through a 3x3 layer 175 / 59 / 82, the dilated 512-channel layer 111 / 52 / 78; with every tile twice 29, 238 and 172.)
// A row in range has the factor 1 in both passes, so its result does not depend on its neighbours.  Filters get their factor
// when they are packed, which costs nothing then, so theirs is 1 in [2^-7, 2^6) only.  Where the packing has seen another factor the
// sums are multiplied before they are stored.
constexpr int kRowShift = 7, kFilterShift = 9; // what a value is multiplied by before it is split, as powers of two
constexpr float kRowUnit = (float)(1 << kRowShift), kFilterUnit = (float)(1 << kFilterShift), kLoScale = 2048.f;
constexpr float kMainUnit = 1.f / (kRowUnit * kFilterUnit), kCrossUnit = kMainUnit / kLoScale; // of the two accumulators
// Biased exponents in range, [low, top]
constexpr uint32_t kRowLow = 127 - 12, kRowTop = 127 + 14 - kRowShift, kFilterLow = 127 - 7, kFilterTop = 127 + 14 - kFilterShift;
__device__ __forceinline__ uint32_t row_exponent(float top) { // biased exponent of a non-negative number, 0 for zero alone
    const uint32_t b = __float_as_uint(top);
    return b ? max(b >> 23, 1u) : 0u;
}
// (zero, infinity and NaN count as in range)
template <uint32_t LOW = kRowLow, uint32_t TOP = kRowTop> __device__ __forceinline__ bool row_out_of_range(uint32_t e) {
    return e - 1u < LOW - 1u || e - (TOP + 1u) < 254u - TOP;
}
template <uint32_t LOW = kRowLow, uint32_t TOP = kRowTop> __device__ __forceinline__ uint32_t row_scale_bits(uint32_t e) { // takes the largest to the top
    return row_out_of_range<LOW, TOP>(e) ? min(127u + TOP - e, 244u) : 127u; // (244: times the unit it is still a float)
}
__device__ __forceinline__ float row_scale(uint32_t e) { return __uint_as_float(row_scale_bits(e) << 23); }
__device__ __forceinline__ float row_unscale(uint32_t e) { return __uint_as_float((254u - row_scale_bits(e)) << 23); }
__device__ __forceinline__ bool filter_out_of_range(uint32_t e) { return row_out_of_range<kFilterLow, kFilterTop>(e); }
__device__ __forceinline__ float filter_unscale(uint32_t e) { return __uint_as_float((254u - row_scale_bits<kFilterLow, kFilterTop>(e)) << 23); }
// A sum times the factors of its row and of its filter, each given as two powers of two of half its exponent: the product of two
// whole factors may be infinite (a zero sum would become NaN) or zero where the sum's own result is neither.  (The first pass stores
// rows in range only, whose factor is 1: there a sum is multiplied by its filter's alone.)
__device__ __forceinline__ float2 factor_halves(float factor) {
    const uint32_t e = __float_as_uint(factor) >> 23, h = (e + 127u) >> 1;
    return make_float2(__uint_as_float(h << 23), __uint_as_float((e + 127u - h) << 23));
}
__device__ __forceinline__ float unscaled(float sum, float2 row, float2 filter) { return sum * (row.x * filter.x) * (row.y * filter.y); }

// Operands of one tile row, eight 32-bit words at a time (a K stage is four such pieces: 32 TF32 values, or 64 halves in pairs),
// split into hi/lo parts — TF32: hi = top 19 bits, lo = x - hi, one value per word; bf16: hi = bf16(x), lo = bf16(x - hi), two
// values per word, the lower K index in the low half; a single pass rounds instead.
// (A stage is 200 to 300 instructions that every transform warp fetches again for every stage — the SM quarter's first-level
// instruction cache does not hold them — at about five cycles each, which is what bounds narrow tiles.  As a rolled loop of
// eight elements it was no faster: the branches and the shorter runs of independent loads cost what the fetches did.)
// fp16: y = x * 2^7, hi = half(y), lo = half((y - hi) * 2^11) (see row_exponent); the accumulators are scaled back when they join.  `top`
// follows the largest magnitude.  (The remainder as a multiply-add that takes the half as it is, instead of a conversion and a packed
// multiply-add: a 128-filter 3x3 layer at batch 64 53.3 -> 52.8 us, a 512-channel one 53.9 -> 52.8.)
template <int PASSES> __device__ __forceinline__ void split_words(const float *v, uint32_t *hi, uint32_t *lo, [[maybe_unused]] float &top) {
    if (PASSES == kMathF16x3) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float2 x = make_float2(v[2 * i], v[2 * i + 1]), y = ptx::mul_f32x2(x, kRowUnit);
            top = ptx::max3_abs(top, x.x, x.y);
            const uint32_t h = ptx::pack_f16x2(y.x, y.y);
            const float2 d = ptx::minus_2048_halves(ptx::mul_f32x2(x, kRowUnit * kLoScale), h);
            hi[i] = h;
            lo[i] = ptx::pack_f16x2(d.x, d.y);
        }
    } else if (PASSES == kMathBf16x3) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t h = ptx::pack_bf16x2(v[2 * i], v[2 * i + 1]);
            hi[i] = h;
            lo[i] = ptx::pack_bf16x2(v[2 * i] - __uint_as_float(h << 16), v[2 * i + 1] - __uint_as_float(h & 0xffff0000u));
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (PASSES == kMathTf32x3) {
                hi[i] = __float_as_uint(v[i]) & 0xffffe000u;
                lo[i] = __float_as_uint(v[i] - __uint_as_float(hi[i]));
            } else { // single pass: round to nearest TF32 instead of letting the tensor core truncate
                hi[i] = ptx::cvt_rna_tf32(v[i]);
            }
        }
    }
}

// Eight consecutive K elements of one tile row.  Where they come from:
//   kGatherTable   im2col through the offset table of the stage (`ko`: the eight entries);
//   kGatherFlat    the same for unpadded whole-plane raw tiles: entries < 0 mean no such element, the filter tap sits in bits
//                  24..30 and `tmask` tells which taps fall inside the input for this pixel;
//   kGatherStride  chunks of a multiple of eight channels: the eight are consecutive channels of ONE tap, `cstride` floats
//                  apart from the first one's table entry - one table read, no per-element tests (kGatherPlain: chunks of a
//                  multiple of 32 channels, one read per stage);
//   kGatherKMajor  matmul with row-major A: half of a 128-byte row piece of the swizzled [128][32] tile (`krow`, 16-byte chunks
//                  c and c + 1).
enum { kGatherTable = 0, kGatherFlat = 1, kGatherStride = 2, kGatherPlain = 3, kGatherKMajor = 4, kGatherBand = 5 };
template <int MODE>
__device__ __forceinline__ void gather8(const int *ko, const float *raw, const uint8_t *krow, int c, int p, uint32_t tmask, int cstride, bool flat,
                                        const float *zero_word, float *v) {
    if (MODE == kGatherKMajor) { // 16-byte chunk c of row p sits at c ^ (p & 7)
        const float4 a = *reinterpret_cast<const float4 *>(krow + ((c ^ (p & 7)) << 4)), b = *reinterpret_cast<const float4 *>(krow + (((c + 1) ^ (p & 7)) << 4));
        v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
    } else if (MODE == kGatherStride) {
        const int o0 = *ko;
        // past the end of the chunk's K range, or a tap outside the input for this pixel: read zeros
        const bool off = o0 < 0 || (flat && !((tmask >> (o0 >> 24)) & 1u));
        const float *q = off ? zero_word : raw + (flat ? (o0 & 0xffffff) : o0);
        const int cs = off ? 0 : cstride;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            v[i] = q[i * cs];
    } else {
        const int4 a = *reinterpret_cast<const int4 *>(ko), b = *reinterpret_cast<const int4 *>(ko + 4);
        const int o[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (MODE == kGatherFlat)
                v[i] = (o[i] >= 0 && ((tmask >> (o[i] >> 24)) & 1u)) ? raw[o[i] & 0xffffff] : 0.f;
            else
                v[i] = raw[o[i]]; // plain table mode has no negative entries
        }
    }
}

// GBMML's operand: row i of the tile meets key k through the band entry p[i][k - i + w].  A chunk is the entries of 64 keys (two K
// stages) for the tile's 128 rows.  A row's entries are contiguous, but rows are 2w + 1 words apart (odd), so each starts
// somewhere else in its first 16 bytes: the transform warps fetch 16-byte pieces from the boundary below (16 lanes per row,
// asynchronous copies, up to three chunks ahead), rows sit kBandPitch words apart in shared memory (16-byte reads of eight
// neighbouring rows then hit different banks), and the thread that owns a row shifts its values into place while it reads
// them.  What lies outside the band, the rows or the sequence counts as zero, whatever the memory holds.  (At n = 10000,
// w = 1000 one 4-byte copy per entry took 66 us: 64 copies and reads with their own addresses and tests per thread and stage,
// which overran the instruction cache as well; a bulk copy per row took 93 us, about 53 cycles of the copy engine each.)
constexpr int kBandStages = 2, kBandKeys = kBandStages * kStageK, kBandPitch = kBandKeys + 4;
// Word of the whole band at which row i's entry for key k0 sits (k0 a multiple of 4), and its place in its 16 bytes.
__device__ __forceinline__ long long band_word(const IgemmParams &P, int zb, int i, int k0) {
    return ((long long)zb * P.m_rows + i) * (2 * P.band_w + 1) + (k0 - i + P.band_w);
}
// One chunk, transform warp `wi` of eight: rows 2 * wi + (lane >> 4), + 16, ..  Sixteen rows on, a row's chunk starts exactly 32w
// words further, so inside the band (all but the first and last chunks of a row tile) the copies need no tests and one
// addition each.  Every lane arrives on `bar` when its copies have landed.
__device__ __forceinline__ void band_copy(const IgemmParams &P, int zb, int i0, int k0, int wi, int lane, uint32_t raw_addr, uint64_t *bar) {
    const int bw = 2 * P.band_w + 1, rows = min(kTileM, P.m_rows - i0), off0 = k0 - i0 + P.band_w;
    const long long row0 = ((long long)zb * P.m_rows + i0) * bw; // first entry of the tile's first row
    const float *base = P.band_p + (row0 & ~3ll);                // word offsets below are relative to this
    const int in0 = (int)(row0 & 3), p0 = 2 * wi + (lane >> 4), c = 4 * (lane & 15);
    const int a0 = (in0 + p0 * bw + off0 - p0) & ~3; // the first row's first word
    uint32_t dst = raw_addr + (uint32_t)(p0 * kBandPitch + c) * 4u;
    // the 17th pieces: one of this warp's sixteen rows per lane
    const int p17 = 2 * wi + (lane & 1) + 16 * ((lane & 15) >> 1);
    const int a17 = ((in0 + p17 * bw + off0 - p17) & ~3) + kBandKeys;
    const uint32_t dst17 = raw_addr + (uint32_t)(p17 * kBandPitch + kBandKeys) * 4u;
    if (rows == kTileM && off0 - (kTileM - 1) >= 0 && off0 + kBandPitch + 3 <= bw) {
        const float *src = base + (a0 + c);
#pragma unroll
        for (int r = 0; r < 8; ++r, src += 32 * P.band_w, dst += 16 * kBandPitch * 4)
            ptx::cp_async_16(dst, src);
        if (lane < 16)
            ptx::cp_async_16(dst17, base + a17);
    } else {
        const int end = (int)min(P.band_words / 4 * 4 - (row0 & ~3ll), 1ll << 30);
        // 16-byte pieces that hold entries of the row (the last, incomplete one of the whole band is left out: with w >= 3 its
        // keys lie past the sequence)
        auto exists = [&](int p, int a) {
            const int row = in0 + p * bw;
            return p < rows && a >= (row & ~3) && a < min((row + bw + 3) & ~3, end);
        };
#pragma unroll 2
        for (int r = 0; r < 8; ++r, dst += 16 * kBandPitch * 4)
            if (exists(p0 + 16 * r, a0 + c + r * 32 * P.band_w))
                ptx::cp_async_16(dst, base + (a0 + c + r * 32 * P.band_w));
        if (lane < 16 && exists(p17, a17))
            ptx::cp_async_16(dst17, base + a17);
    }
    ptx::cp_async_mbar_arrive_noinc(bar);
}
// Eight of a row's operands: `src` is their place in shared memory, `shift` the row's place in its first 16 bytes, [lo_e, hi_e)
// the elements that exist.
__device__ __forceinline__ void band_take8(const float *src, int shift, int lo_e, int hi_e, float *v) {
    float q[12];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float4 t = *reinterpret_cast<const float4 *>(src + 4 * c);
        q[4 * c] = t.x, q[4 * c + 1] = t.y, q[4 * c + 2] = t.z, q[4 * c + 3] = t.w;
    }
#pragma unroll
    for (int e = 0; e < 11; ++e)
        q[e] = (shift & 1) ? q[e + 1] : q[e];
#pragma unroll
    for (int e = 0; e < 8; ++e)
        v[e] = e >= lo_e && e < hi_e ? ((shift & 2) ? q[e + 2] : q[e]) : 0.f;
}

// Split-K reduction inside a thread-block cluster.  The ksplit CTAs of one output tile form a cluster; CTA `rank` owns
// BN/ksplit columns of the tile, and every CTA has pushed its partial sums of those columns into this CTA's shared memory
// as [source rank][column][pixel].  A thread adds the ksplit copies of an element in rank order (the sum does not depend
// on timing) and stores act(sum + bias).
template <int ACT>
__device__ __forceinline__ void cluster_reduce_store(const float *stage, int ksplit, int rank, int cols, int et /*0..255*/,
                                                     int f_tile0, int Fg, const float *bias, const float *rp, float *yp /*this pixel, filter 0*/,
                                                     long long ys_f, bool vec_ok) {
    const int px = et & (kTileM - 1), half = et >> 7;
    if (vec_ok) {
        // Filters are contiguous in y (row-major matmul output): a thread owns a run of cols/2 consecutive columns of its
        // pixel and stores them 16 bytes at a time; with the interleaved assignment below every 4-byte store would
        // touch its own 32-byte sector.
        const int run = cols >> 1; // 2, 4, 8, ... 32
        for (int c0 = half * run; c0 < (half + 1) * run; c0 += 4) {
            const int f = f_tile0 + rank * cols + c0, nv = min(4, run);
            if (f >= Fg)
                break;
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
            // (kept as a loop: this code runs once per CTA, straight out of a cold instruction cache, so its length is its cost)
            const float *sp = stage + c0 * kTileM + px;
#pragma unroll 1
            for (int r = 0; r < ksplit; ++r, sp += cols * kTileM)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (j < nv)
                        acc[j] += sp[j * kTileM]; // rank order for every element
            if (nv == 4) { // Fg % 4 == 0 and f % 4 == 0 here: the whole quad is inside the row, and 16-byte aligned in y / residual
                if (bias != nullptr) {
                    float4 b;
                    if ((reinterpret_cast<uintptr_t>(bias) & 15) == 0)
                        b = __ldg(reinterpret_cast<const float4 *>(bias + f));
                    else
                        b = make_float4(__ldg(bias + f), __ldg(bias + f + 1), __ldg(bias + f + 2), __ldg(bias + f + 3));
                    acc[0] += b.x, acc[1] += b.y, acc[2] += b.z, acc[3] += b.w;
                }
                if (rp != nullptr) {
                    const float4 r4 = __ldg(reinterpret_cast<const float4 *>(rp + f));
                    acc[0] += r4.x, acc[1] += r4.y, acc[2] += r4.z, acc[3] += r4.w;
                }
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    acc[j] = act_fn<ACT>(acc[j]);
                *reinterpret_cast<float4 *>(yp + f) = make_float4(acc[0], acc[1], acc[2], acc[3]);
            } else {
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    if (bias != nullptr)
                        acc[j] += __ldg(bias + f + j);
                    if (rp != nullptr)
                        acc[j] += __ldg(rp + f + j);
                    acc[j] = act_fn<ACT>(acc[j]);
                }
                *reinterpret_cast<float2 *>(yp + f) = make_float2(acc[0], acc[1]);
            }
        }
        return;
    }
#pragma unroll 2
    for (int cl = half; cl < cols; cl += 2) {
        const int f = f_tile0 + rank * cols + cl;
        if (f >= Fg)
            break;
        const float *sp = stage + cl * kTileM + px;
        float acc = sp[0]; // rank order, as in the 16-byte path
#pragma unroll 1
        for (int r = 1; r < ksplit; ++r)
            acc += sp[r * cols * kTileM];
        if (bias != nullptr)
            acc += __ldg(bias + f);
        if (rp != nullptr)
            acc += __ldg(rp + (long long)f * ys_f);
        yp[(long long)f * ys_f] = act_fn<ACT>(acc);
    }
}

// Drain warps: a thread keeps the BN sums of its tile row in registers.  add_main: sums (+)= main accumulator; with the cross
// terms on top for the last (or only) group of a tile: hi*hi sum + (lo*hi + hi*lo) sum, one rounded fp32 add.
template <int PASSES> __device__ __forceinline__ float join_sums(uint32_t main_sum, uint32_t cross_sum) {
    if (PASSES == kMathF16x3)
        return fmaf(__uint_as_float(cross_sum), kCrossUnit, __uint_as_float(main_sum) * kMainUnit);
    return PASSES != kMathTf32x1 ? __uint_as_float(main_sum) + __uint_as_float(cross_sum) : __uint_as_float(main_sum);
}
template <int PASSES, bool CROSS>
__device__ __forceinline__ void drain_add(float (&racc)[128], uint32_t tmain, uint32_t tcross, int BN, bool first) {
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        if (b * 16 < BN) {
            uint32_t v[16], c[16];
            ptx::tmem_ld_32x16(tmain + (uint32_t)(b * 16), v);
            if (CROSS)
                ptx::tmem_ld_32x16(tcross + (uint32_t)(b * 16), c);
            ptx::tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                float x = __uint_as_float(v[j]);
                if (!first)
                    x = racc[b * 16 + j] + x;
                racc[b * 16 + j] = CROSS ? join_sums<PASSES>(__float_as_uint(x), c[j]) : x;
            }
        }
    }
}

// One 32-column block of a warp's 32 tile rows, sums in r (thread = row), to y, through the warp's 4 KB block of shared memory where
// that makes the stores coalesced:
//   kStorePixels  pixels contiguous in y (NCHW), 16-byte aligned: a lane stores four pixels of one filter;
//   kStoreFilters filters contiguous in y (row-major matmul, channels last), aligned: a lane stores four filters of one row;
//   kStoreRows    the same off the 16-byte grid: a store instruction writes 32 filters of one row;
//   kStoreAny     anything else: every thread stores its own row (for NCHW off the grid that is 32 pixels of one filter).
// Straight-line code with predicated loads and stores: a tile's successor lasts only two to four thousand cycles at 64 filters,
// and a taken branch costs 70 to 250 of them (see the MMA issuer; as a loop with tests per store a tile took 15000).  For the
// same reason the long activations are a loop of their own over the block in shared memory, with bias and residual.
enum { kStorePixels = 0, kStoreFilters = 1, kStoreRows = 2, kStoreAny = 3 };
struct StoreJob {
    float *y;                // filter 0 of the group
    const float *bias, *res; // the same, or null
    long long ys_f, y_off, y_off0; // this row, the warp's first row
    int Fg, act, nvalid, lane;
    bool valid;
};
// fp16, rare: a block's sums times the factors of the filters and, in the second pass, that of the row.
template <bool SECOND> __device__ __forceinline__ void unscale_block(float *r, float unscale, const float *fscale, int f0, int Fg, bool factors, int lane) {
    const float mine = factors && f0 + lane < Fg ? __ldg(fscale + f0 + lane) : 1.f;
    if constexpr (SECOND) {
        const float2 row = factor_halves(unscale), filter = factor_halves(mine);
#pragma unroll
        for (int j = 0; j < 32; ++j)
            r[j] = unscaled(r[j], row, make_float2(__shfl_sync(0xffffffffu, filter.x, j), __shfl_sync(0xffffffffu, filter.y, j)));
    } else {
#pragma unroll
        for (int j = 0; j < 32; ++j)
            r[j] *= __shfl_sync(0xffffffffu, mine, j);
    }
}
template <bool RES>
__device__ __forceinline__ void store_pixels(const StoreJob &J, const float *bias, const float *stage, int f0) { // four pixels that are all valid per lane
    const int px = (J.lane & 7) * 4, cq = J.lane >> 3, fmax = px + 4 <= J.nvalid ? J.Fg - f0 - cq : 0; // filters left from this lane's first one
    const long long off = J.y_off0 + (long long)(f0 + cq) * J.ys_f + px, step = 4 * J.ys_f;
    float4 v[8];
    if (RES) {
        const float *rs = J.res + off;
#pragma unroll
        for (int i = 0; i < 8; ++i, rs += step)
            v[i] = 4 * i < fmax ? __ldg(reinterpret_cast<const float4 *>(rs)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float b[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
        b[i] = bias != nullptr && 4 * i < fmax ? __ldg(bias + f0 + cq + 4 * i) : 0.f;
    float *dst = J.y + off;
#pragma unroll
    for (int i = 0; i < 8; ++i, dst += step) {
        float4 q = *reinterpret_cast<const float4 *>(stage + (cq + 4 * i) * 32 + px);
        if (bias != nullptr)
            q.x += b[i], q.y += b[i], q.z += b[i], q.w += b[i];
        if (RES) // y = act(sum + bias + residual): the residual's four pixels sit where y's will
            q.x += v[i].x, q.y += v[i].y, q.z += v[i].z, q.w += v[i].w;
        if (J.act == PETB200_ACT_RELU)
            q.x = fmaxf(q.x, 0.f), q.y = fmaxf(q.y, 0.f), q.z = fmaxf(q.z, 0.f), q.w = fmaxf(q.w, 0.f);
        if (4 * i < fmax)
            *reinterpret_cast<float4 *>(dst) = q;
    }
}
// kStoreFilters / kStoreRows / kStoreAny; the block (filters, rows) lies in `stage`, for kStoreAny in r.  RES: with a residual (a test
// per store would be a branch per store).
template <bool RES>
__device__ __forceinline__ void store_filters(const StoreJob &J, const float *bias, const float *stage, int f0) {
    const int lane = J.lane, c = lane & 7, f = f0 + 4 * c;
    const bool live = f < J.Fg, relu = J.act == PETB200_ACT_RELU; // (Fg % 4 == 0 in this mode)
    float4 bv = make_float4(0.f, 0.f, 0.f, 0.f);
    if (bias != nullptr && live)
        bv = make_float4(__ldg(bias + f), __ldg(bias + f + 1), __ldg(bias + f + 2), __ldg(bias + f + 3));
    const long long yo = J.valid ? J.y_off : -1;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int row = 4 * i + (lane >> 3);
        const long long off = __shfl_sync(0xffffffffu, yo, row);
        const bool go = off >= 0 && live;
        float4 v = *reinterpret_cast<const float4 *>(stage + row * 32 + ((c ^ (row & 7)) << 2));
        v.x += bv.x, v.y += bv.y, v.z += bv.z, v.w += bv.w;
        if (RES) {
            const float4 q = go ? __ldg(reinterpret_cast<const float4 *>(J.res + off + f)) : make_float4(0.f, 0.f, 0.f, 0.f);
            v.x += q.x, v.y += q.y, v.z += q.z, v.w += q.w;
        }
        if (relu)
            v.x = fmaxf(v.x, 0.f), v.y = fmaxf(v.y, 0.f), v.z = fmaxf(v.z, 0.f), v.w = fmaxf(v.w, 0.f);
        if (go)
            *reinterpret_cast<float4 *>(J.y + off + f) = v;
    }
}
// Rows a constant pitch apart (a matmul's, or pixels of one image) take one pointer that moves down them, which is half the
// instructions of an offset per row (29 x 78 x 662 x 24: 24.6 -> 22 us, 4 x 500 x 1001 x 768: 19.6 -> 18.4 us).
template <bool RES>
__device__ __forceinline__ void store_rows(const StoreJob &J, const float *bias, const float *stage, int f0) {
    const int lane = J.lane, f = f0 + lane;
    const bool live = f < J.Fg, relu = J.act == PETB200_ACT_RELU;
    const float bv = bias != nullptr && live ? __ldg(bias + f) : 0.f;
    const long long pitch = __shfl_sync(0xffffffffu, J.y_off, 1) - J.y_off0;
    if (__all_sync(0xffffffffu, J.valid == (lane < J.nvalid) && (!J.valid || J.y_off == J.y_off0 + lane * pitch))) {
        const int rows = live ? J.nvalid : 0;
        float *dst = J.y + J.y_off0 + f;
        const float *rs = RES ? J.res + J.y_off0 + f : nullptr;
#pragma unroll
        for (int row = 0; row < 32; ++row, dst += pitch) {
            float v = stage[row * 32 + (lane ^ row)] + bv;
            if (RES) {
                v += row < rows ? __ldg(rs) : 0.f;
                rs += pitch;
            }
            v = relu ? fmaxf(v, 0.f) : v;
            if (row < rows)
                *dst = v;
        }
        return;
    }
    const long long yo = J.valid ? J.y_off : -1;
#pragma unroll 1
    for (int row = 0; row < 32; ++row) {
        const long long off = __shfl_sync(0xffffffffu, yo, row);
        const bool go = off >= 0 && live;
        float v = stage[row * 32 + (lane ^ row)] + bv;
        if (RES)
            v += go ? __ldg(J.res + off + f) : 0.f;
        v = relu ? fmaxf(v, 0.f) : v;
        if (go)
            J.y[off + f] = v;
    }
}
template <bool RES, int AHEAD /*values of the residual in flight*/>
__device__ __forceinline__ void store_any(const StoreJob &J, const float *bias, const float *r, int f0) {
    const int nf = J.valid ? J.Fg - f0 : 0; // filters of this thread's row
    const bool relu = J.act == PETB200_ACT_RELU;
    const float bv = bias != nullptr && f0 + J.lane < J.Fg ? __ldg(bias + f0 + J.lane) : 0.f; // lane j holds filter j's
    float *dst = J.y + J.y_off + (long long)f0 * J.ys_f;
    const float *rs = RES ? J.res + J.y_off + (long long)f0 * J.ys_f : nullptr;
    if constexpr (AHEAD == 1) {
#pragma unroll
        for (int j = 0; j < 32; ++j, dst += J.ys_f) {
            float v = r[j] + __shfl_sync(0xffffffffu, bv, j);
            if (RES)
                v += j < nf ? __ldg(rs + (long long)j * J.ys_f) : 0.f;
            if (j < nf)
                *dst = relu ? fmaxf(v, 0.f) : v;
        }
    } else {
#pragma unroll
        for (int j = 0; j < 32; j += AHEAD) {
            float q[AHEAD];
#pragma unroll
            for (int i = 0; i < AHEAD; ++i)
                q[i] = RES && j + i < nf ? __ldg(rs + (long long)(j + i) * J.ys_f) : 0.f;
#pragma unroll
            for (int i = 0; i < AHEAD; ++i, dst += J.ys_f) {
                float v = r[j + i] + __shfl_sync(0xffffffffu, bv, j + i);
                if (RES)
                    v += q[i];
                if (j + i < nf)
                    *dst = relu ? fmaxf(v, 0.f) : v;
            }
        }
    }
}
// This thread's row through one of the long activations, with bias and residual.  One warp per SM quarter stores, so this is a chain of
// latencies (shared memory, exponential, reciprocal): eight filters at a time, and the choice of activation outside the loop.
// Four at a time with the choice inside, a 3x3 convolution of 18 x 16 x 24 x 24 to 216 filters took 42.8 us with a sigmoid, 33.0 with
// GELU, 30.8 with tanh and 15.2 with none; now 36.6 (its division), 24.6, 22.6 and 13.6.
template <int ACT>
__device__ __forceinline__ void activate_row(const StoreJob &J, float *stage, const float *rp, float bias, int f0) {
#pragma unroll 1
    for (int j = 0; j < 32 && f0 + j < J.Fg; j += 8) {
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
            v[i] = stage[(j + i) * 32 + J.lane] + __shfl_sync(0xffffffffu, bias, j + i);
        if (rp != nullptr) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (f0 + j + i < J.Fg)
                    v[i] += __ldg(rp + (long long)(j + i) * J.ys_f);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
            stage[(j + i) * 32 + J.lane] = act_fn<ACT>(v[i]);
    }
}
__device__ __forceinline__ void activate_block(const StoreJob &J, float *r, float *stage, int f0) {
    const int lane = J.lane;
#pragma unroll
    for (int j = 0; j < 32; ++j)
        stage[j * 32 + lane] = r[j];
    const float *rp = J.res != nullptr && J.valid ? J.res + J.y_off + (long long)f0 * J.ys_f : nullptr;
    const float bias = J.bias != nullptr && f0 + lane < J.Fg ? __ldg(J.bias + f0 + lane) : 0.f; // lane j holds filter j's
    if (J.act == PETB200_ACT_SIGMOID)
        activate_row<PETB200_ACT_SIGMOID>(J, stage, rp, bias, f0);
    else if (J.act == PETB200_ACT_TANH)
        activate_row<PETB200_ACT_TANH>(J, stage, rp, bias, f0);
    else
        activate_row<PETB200_ACT_GELU>(J, stage, rp, bias, f0);
#pragma unroll
    for (int j = 0; j < 32; ++j)
        r[j] = stage[j * 32 + lane];
    __syncwarp();
}
// LONG: with one of the long activations (RES is then false, activate_block adds a residual).  Its own instances: beside the others'
// code it cost ResNet-18 at batch 64 5 %, whose layers have none of it.
// AHEAD: 8 where the thread keeps a row of 128 sums (left to the compiler the loads were waited for one by one there: 46 x 116 x 19 x 19 to
// 299 filters 108 us, now 59); elsewhere the compiler moves them up itself (eight: 2 x 16 x 63 x 63 to 142 filters 13.9 -> 15.9, 32: 16.5).
template <int MODE, bool RES, bool LONG, int AHEAD>
__device__ __forceinline__ void store_block(const StoreJob &J, float *r /*32 sums*/, float *stage, int f0) {
    const int lane = J.lane;
    __syncwarp(); // the previous block has been read
    if constexpr (LONG) {
        activate_block(J, r, stage, f0);
        StoreJob R = J; // bias and residual have been added
        R.bias = R.res = nullptr, R.act = PETB200_ACT_NONE;
        store_block<MODE, false, false, AHEAD>(R, r, stage, f0);
        return;
    }
    const float *bias = J.bias;
    if (MODE == kStorePixels) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
            stage[j * 32 + lane] = r[j];
        __syncwarp();
        store_pixels<RES>(J, bias, stage, f0);
        if (__builtin_expect((J.nvalid & 3) != 0, 0)) { // the last one to three pixels of a ragged window are left
            if (J.valid && lane >= (J.nvalid & ~3)) {
                const long long off = J.y_off + (long long)f0 * J.ys_f;
#pragma unroll 1
                for (int j = 0; j < 32 && f0 + j < J.Fg; ++j) {
                    float v = stage[j * 32 + lane] + (bias != nullptr ? __ldg(bias + f0 + j) : 0.f);
                    if (RES)
                        v += __ldg(J.res + off + j * J.ys_f);
                    J.y[off + j * J.ys_f] = J.act == PETB200_ACT_RELU ? fmaxf(v, 0.f) : v;
                }
            }
        }
    } else if (MODE == kStoreFilters) {
        // row r of the block at [r][32], 16-byte chunk c at c ^ (r & 7): conflict-free both ways
#pragma unroll
        for (int c = 0; c < 8; ++c)
            *reinterpret_cast<float4 *>(stage + lane * 32 + ((c ^ (lane & 7)) << 2)) = make_float4(r[4 * c], r[4 * c + 1], r[4 * c + 2], r[4 * c + 3]);
        __syncwarp();
        store_filters<RES>(J, bias, stage, f0);
    } else if (MODE == kStoreRows) { // word c of row r at c ^ r
#pragma unroll
        for (int j = 0; j < 32; ++j)
            stage[lane * 32 + (j ^ lane)] = r[j];
        __syncwarp();
        store_rows<RES>(J, bias, stage, f0);
    } else {
        store_any<RES, AHEAD>(J, bias, r, f0);
    }
}
// f(mode, with residual, long activation) as compile-time constants: the loops around store_block are instantiated per way of storing.
template <typename F> __device__ __forceinline__ void with_store_mode(int mode, bool res, int act, F &&f) {
    const std::integral_constant<bool, true> yes;
    const std::integral_constant<bool, false> no;
    auto pick = [&](auto mode_c) {
        if (__builtin_expect(act > PETB200_ACT_RELU, 0))
            f(mode_c, no, yes);
        else
            res ? f(mode_c, yes, no) : f(mode_c, no, no);
    };
    if (mode == kStorePixels)
        pick(std::integral_constant<int, kStorePixels>());
    else if (mode == kStoreFilters)
        pick(std::integral_constant<int, kStoreFilters>());
    else if (mode == kStoreRows)
        pick(std::integral_constant<int, kStoreRows>());
    else
        pick(std::integral_constant<int, kStoreAny>());
}

// A set of barriers (the last one is a word in each of the roles' slots, see the kernel).
__device__ __forceinline__ void init_barriers(uint64_t *bars, int raw_arrivals) {
    uint64_t *raw_full = bars, *raw_empty = bars + kMaxNR, *b_full = bars + 2 * kMaxNR, *b_empty = b_full + kMaxNB;
    uint64_t *a_full = b_empty + kMaxNB, *a_empty = a_full + 4, *acc_full = a_empty + 4;
    for (int i = 0; i < kMaxNR; ++i) {
        ptx::mbar_init(raw_full + i, raw_arrivals);
        ptx::mbar_init(raw_empty + i, 8);
    }
    for (int i = 0; i < kMaxNB; ++i) {
        ptx::mbar_init(b_full + i, 1);
        ptx::mbar_init(b_empty + i, 1);
    }
    for (int i = 0; i < kNA; ++i) {
        ptx::mbar_init(a_full + i, 4);
        ptx::mbar_init(a_empty + i, 1);
    }
    ptx::mbar_init(acc_full, 1);
    ptx::mbar_init(acc_full + 4, 1); // acc_ready
    ptx::mbar_init(acc_full + 5, 4); // flushed
    ptx::mbar_init(acc_full + 6, 1); // acc_full1
    ptx::mbar_init(acc_full + 7, 4); // acc_empty
    ptx::mbar_init(acc_full + 8, 4);
    ptx::mbar_init(acc_full + 9, 1);  // trash
    ptx::mbar_init(acc_full + 10, 8); // scanned
}

// What lies where in a CTA's shared memory.
struct CtaSmem {
    uint8_t *smem, *sB, *sRaw;
    int *sKoff;
    float *sSplit;
    long long *sYoff; // split-K only: each tile row's offset in y
    uint64_t *bars;   // (the barriers are named where they are used)
    // words that share the first set of barriers' block
    uint32_t *tmem_slot;
    volatile int *abort_flag;
    float *zero_word;        // holds 0.0f: what a masked-off filter tap reads
    volatile int *left_over; // fp16: rows were out of range, a second pass is needed
    uint8_t *row_exps;       // fp16: [kExpSlots][set][row]
    __device__ __forceinline__ CtaSmem(uint8_t *base, const IgemmParams &P) : smem(base) {
        const SmemLayout &L = P.L;
        sB = smem + L.b_off;
        sRaw = smem + L.raw_off;
        sKoff = reinterpret_cast<int *>(smem + L.koff_off);
        sSplit = reinterpret_cast<float *>(smem + L.split_off);
        sYoff = reinterpret_cast<long long *>(smem + L.split_off + 512u * (uint32_t)P.BN);
        bars = reinterpret_cast<uint64_t *>(smem + L.bar_off);
        uint64_t *words = bars + 2 * kMaxNR + 2 * kMaxNB + 8;
        tmem_slot = reinterpret_cast<uint32_t *>(words + 1);
        abort_flag = reinterpret_cast<volatile int *>(words + 2);
        zero_word = reinterpret_cast<float *>(words + 3);
        left_over = reinterpret_cast<volatile int *>(words + 11);
        row_exps = smem + L.exp_off;
    }
};
// Filter tile, part of K and group or batch entry of a CTA with one tile.
struct CtaPlace {
    int ntile = 0, ksp = 0, zb = 0;
    __device__ __forceinline__ CtaPlace(int pp, const IgemmParams &P) {
        if (!pp) {
            ntile = (int)blockIdx.y >> P.ks_log;
            ksp = (int)blockIdx.y & (P.ksplit - 1);
            zb = (int)blockIdx.z;
        }
    }
};
constexpr uint32_t kTmemCols = 512;

// One pass over the CTA's tiles, by role.  fp16 may need a second, whose items may be every tile twice (see row_exponent).
// BAND: 0 ordinary operands; 1 G2BMM (banded epilogue, key windows per tile; persistent row-major mode only); 2 GBMML (A operand
// gathered from the band in global memory; row-major mode only).  Kernels of their own, so that the others carry none of it.
template <bool A_KMAJOR, int PASSES, int PP, int BAND, bool SECOND>
__device__ __forceinline__ void igemm_pass(const CUtensorMap &tmap_x, const CUtensorMap &tmap_bhi, const CUtensorMap &tmap_blo, const IgemmParams &P,
                                           const CtaSmem &S, const uint32_t tmem_base, const CtaPlace &at) {
    constexpr int pass = SECOND ? 1 : 0;
    const SmemLayout &L = P.L;
    uint8_t *const smem = S.smem, *const sB = S.sB, *const sRaw = S.sRaw;
    int *const sKoff = S.sKoff;
    float *const sSplit = S.sSplit, *const zero_word = S.zero_word;
    long long *const sYoff = S.sYoff;
    volatile int *const abort_flag = S.abort_flag, *const left_over = S.left_over;
    uint8_t *const row_exps = S.row_exps;
    uint64_t *const bars = S.bars + pass * (kBarBytes / 8);
    const std::integral_constant<bool, SECOND> second_c;

    constexpr bool SPLIT = PASSES != kMathTf32x1; // hi/lo operands, two accumulators
    constexpr bool REDO = PASSES == kMathF16x3;   // rows out of range take a second pass (see row_exponent)
    constexpr bool HALF = PASSES == kMathBf16x3 || PASSES == kMathF16x3;
    constexpr int KE = HALF ? 64 : 32;            // K elements per stage
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int ntile = at.ntile, zb = at.zb; // (persistent mode: set per tile by set_tile)
    const int ksp = at.ksp;
    const uint32_t b_half = (uint32_t)P.BN * 128u;
    // TMEM columns: [0,BN) accumulator of the hi*hi products, [BN,2*BN) accumulator of the two small cross terms (persistent
    // narrow tiles: a second such pair behind them), [256,512) the A stages
    constexpr uint32_t kACol = 256;
    constexpr bool two_regions = PP == kNarrow;

    // Tile origin in the input: first image, depth slice, row and (16-byte aligned) column of the raw box.  `bx` is the
    // pixel-tile index: blockIdx.x, or in persistent mode every gridDim.x-th tile from there.
    int bx = (int)blockIdx.x;
    const int ntl = PP ? P.tiles_each + ((int)blockIdx.x < P.tiles_extra ? 1 : 0) : 1; // tiles of this CTA
    int n_lo = 0, q0 = 0, unit0 = 0, z_start = 0, y_start = 0, x_start = 0, w_zl = 0, w_yl = 0, w_tx = 0;
    auto set_tile = [&](int tile) {
        bx = tile;
        if (PP) {
            const int m = P.by_ntiles.div(tile);
            ntile = tile - m * P.ntiles;
            zb = P.by_mtiles.div(m);
            bx = m - zb * P.mtiles;
        }
        n_lo = 0, q0 = 0, unit0 = 0, w_zl = 0, w_yl = 0, w_tx = 0;
        if (A_KMAJOR) {
            z_start = y_start = x_start = 0; // the tile is rows [bx*128, +128) of A[zb]
        } else if (P.wide) {
            const int row = P.by_row_tiles.div(bx), plane = P.by_ohn.div(row);
            w_tx = bx - row * P.row_tiles;
            w_yl = row - plane * P.ohn;
            n_lo = P.by_od.div(plane);
            w_zl = plane - n_lo * P.OD;
            z_start = w_zl * P.sd - P.pd;
            y_start = (P.oh0 + w_yl) * P.sh - P.ph;
            const int xs = (P.ow0 + w_tx * kTileM) * P.sw - P.pw;
            x_start = (xs >= 0) ? (xs & ~3) : -(((-xs) + 3) & ~3);
        } else {
            const int tu = P.by_tpi.div(bx);
            q0 = (bx - tu * P.tpi) * kTileM;
            unit0 = tu * P.ipt;
            n_lo = P.by_od.div(unit0);
            const int yl_lo = P.ipt > 1 ? 0 : P.by_own.div(q0); // first output row of the tile
            z_start = (unit0 - n_lo * P.OD) * P.sd - P.pd;
            y_start = (P.oh0 + yl_lo) * P.sh - P.ph;
            x_start = P.x0;
        }
        if (!A_KMAJOR && P.flat)
            z_start = y_start = x_start = 0; // the raw tile holds whole planes
    };
    set_tile((int)blockIdx.x);
    // Row p of this CTA's tile: is it an output pixel, where does its receptive field start in the raw tile, where does
    // it go in y.
    auto pixel_geom = [&](int p, bool &valid, int &base_p, long long &y_off) {
        base_p = 0;
        y_off = 0;
        if (A_KMAJOR) {
            const int row = bx * kTileM + p;
            valid = row < P.m_rows;
            y_off = (long long)zb * P.ys_n + (long long)row * P.ys_p;
        } else if (P.wide) {
            const int xl = w_tx * kTileM + p;
            valid = xl < P.own;
            if (valid) {
                const int oh = P.oh0 + w_yl, ow = P.ow0 + xl;
                base_p = ow * P.sw - P.pw - x_start;
                const long long img = P.z_is_batch ? (long long)zb : (long long)n_lo;
                y_off = img * P.ys_n + ((long long)(w_zl * P.OH + oh) * P.OW + ow) * P.ys_p;
            }
        } else {
            int ul = 0, q = q0 + p;
            if (P.ipt > 1) {
                ul = P.by_pw.div(p);
                q = p - ul * P.Pw;
            }
            const int unit = unit0 + ul;
            valid = (ul < P.ipt) && (unit < P.units) && (q < P.Pw);
            if (valid) {
                const int n = P.by_od.div(unit);
                const int zl = unit - n * P.OD;
                const int yl = P.by_own.div(q);
                const int xl = q - yl * P.own;
                const int oh = P.oh0 + yl, ow = P.ow0 + xl;
                base_p = (((n - n_lo) * P.BC * P.RD + (zl * P.sd - P.pd - z_start)) * P.RH + (oh * P.sh - P.ph - y_start)) * P.RW +
                         (ow * P.sw - P.pw - x_start);
                const long long img = P.z_is_batch ? (long long)zb : (long long)n;
                y_off = img * P.ys_n + ((long long)(zl * P.OH + oh) * P.OW + ow) * P.ys_p;
            }
        }
    };
    // May runs of pixels be stored 16 bytes at a time?  Pixel-contiguous NCHW output, full-width rows (no column window), one
    // plane per tile, 16-byte aligned runs (of y and of the residual, which is laid out like y).
    auto pixel_runs = [&]() {
        const long long plane_elems = (long long)P.OD * P.OH * P.OW;
        return P.ys_p == 1 && P.ipt == 1 && P.own == P.OW && P.ow0 == 0 && (plane_elems & 3) == 0 && (P.ys_n & 3) == 0 &&
               ((P.OH * P.OW) & 3) == 0 && (!P.wide || (P.OW & 3) == 0) && (P.ys_f & 3) == 0 && ((P.oh0 * P.OW) & 3) == 0 &&
               ((reinterpret_cast<uintptr_t>(P.y) | reinterpret_cast<uintptr_t>(P.res)) & 15) == 0;
    };
    auto store_mode = [&]() -> int {
        const bool filters_run = (P.ys_f == 1) && ((P.ys_p & 3) == 0) && ((P.ys_n & 3) == 0) && ((P.Fg & 3) == 0) &&
                                 (((reinterpret_cast<uintptr_t>(P.y) | reinterpret_cast<uintptr_t>(P.res)) & 15) == 0);
        return pixel_runs() ? kStorePixels : (filters_run ? kStoreFilters : (P.ys_f == 1 ? kStoreRows : kStoreAny));
    };
    // fp16: has some filter of the packed operand a factor other than 1?  Asked by the warps that store before they have anything to
    // store; the answer is waited for where it is used.
    [[maybe_unused]] auto ask_factors = [&]() -> uint32_t {
        uint32_t word = 0;
        if (REDO)
            asm volatile("ld.global.u32 %0, [%1];" : "=r"(word) : "l"(P.factor_word));
        return word;
    };
    [[maybe_unused]] auto any_factor = [&](uint32_t word) -> bool {
        asm volatile("" : "+r"(word));
        return REDO && (word >> 16) == (word & 0xffffu);
    };
    // split-K: this CTA reduces the channel chunks [c0, c1)
    const int c0 = (ksp * P.nchunks) >> P.ks_log, c1 = ((ksp + 1) * P.nchunks) >> P.ks_log;
    const int KS = (c1 - c0) * P.spc;

    if (!SECOND && warp < kSetWarp)
        ptx::reg_dealloc<Regs<PP>::control>();
    // second pass: 1 where every tile is two items, the first for its exponents alone, the second for its sums
    const int twice = SECOND && ntl > kExpSlots ? 1 : 0;
    [[maybe_unused]] auto for_sums = [&](int item) -> bool { return !twice || (item & 1); };
    auto tile_of = [&](int item) { return (int)blockIdx.x + (item >> twice) * (int)gridDim.x; };
    uint64_t *raw_full = bars, *raw_empty = bars + kMaxNR;
    uint64_t *b_full = bars + 2 * kMaxNR, *b_empty = b_full + kMaxNB; // up to kMaxNB stages
    uint64_t *a_full = b_empty + kMaxNB, *a_empty = a_full + 4;       // up to 4 stages
    uint64_t *acc_full = a_empty + 4;
    uint64_t *acc_ready = acc_full + 4; // a group of `fl` K stages has been accumulated: the main accumulator may be drained
    uint64_t *flushed = acc_full + 5;   // the four drain warps have drained it: the MMA warp may restart it
    uint64_t *acc_full1 = acc_full + 6; // persistent mode: the second accumulator region is complete
    uint64_t *acc_empty = acc_full + 7; // [2]: the drain warps have read accumulator region 0 / 1 out
    uint64_t *trash = acc_full + 9;     // takes the MMA thread's releases after it gave up
    [[maybe_unused]] uint64_t *scanned = acc_full + 10; // second pass: both transform sets have recorded a tile's exponents
    const int items = ntl << twice;
    // fp16: exponent of row `row` of a tile (one of a single stage was seen by one set alone; a pair's second item has its first's)
    [[maybe_unused]] auto exponent_of = [&](int item, int row) -> uint32_t {
        if (twice)
            item &= ~1;
        const volatile uint8_t *e = row_exps + ((item >> twice) & (kExpSlots - 1)) * 2 * kTileM + row;
        return KS == 1 ? (uint32_t)e[(item & 1) * kTileM] : max((uint32_t)e[0], (uint32_t)e[kTileM]);
    };
    // Asked by a warp that stores 32 rows, one of them of exponent e: are they stored in this pass?
    [[maybe_unused]] auto store_now = [&](uint32_t e, bool valid) -> bool {
        const bool later = __any_sync(0xffffffffu, valid && row_out_of_range(e));
        if (__builtin_expect(later && pass == 0, 0))
            *left_over = 1;
        return later == SECOND;
    };
    if (warp == 0) {
        // ---------------- packed-weight producer (one thread) ----------------
        if (lane == 0) {
            int sb = 0;
            uint32_t pb = 1; // first pass over the ring: every slot is free
            bool go = true;
            for (int tl = 0; tl < items && go; ++tl) {
                if (PP)
                    set_tile(tile_of(tl));
                int row0 = zb * P.Fg + ntile * P.BN;
                int kx = c0 * P.spc * KE; // first K element of the stage
                if (BAND == 2) // the key window of the row tile, start rounded down to a multiple of 4
                    kx += (bx * kTileM - P.band_w) & ~3;
                if (BAND == 1) // the key window moves with the row tile (rows before the tensor or past it read as zero / are masked)
                    row0 = zb * P.m_rows + bx * kTileM - P.band_w + ntile * P.BN;
                for (int ks = 0; ks < KS; ++ks, kx += KE) {
                    if (!ptx::mbar_wait(b_empty + sb, pb, abort_flag)) {
                        go = false;
                        break;
                    }
                    uint8_t *dst = sB + (size_t)sb * 2 * b_half;
                    ptx::mbar_expect_tx(b_full + sb, (SPLIT ? 2u : 1u) * b_half + (P.starve ? 64u : 0u));
                    ptx::tma_load_2d(dst, &tmap_bhi, b_full + sb, kx, row0);
                    if (SPLIT)
                        ptx::tma_load_2d(dst + b_half, &tmap_blo, b_full + sb, kx, row0);
                    if (++sb == P.NB) {
                        sb = 0;
                        pb ^= 1u;
                    }
                }
            }
        }
    } else if (warp == 2) {
        // ---------------- raw activation producer ----------------
        if (BAND != 2 && lane == 0) { // (GBMML's transform warps fetch their operand themselves)
            const uint32_t bytes = (uint32_t)P.RN * P.BC * P.RD * P.RH * P.RW * 4u;
            int rb = 0;
            uint32_t pr = 1; // first pass over the ring: every buffer is free
            bool go = true;
            for (int tl = 0; tl < items && go; ++tl) {
            if (tl > 0 || pass)
                set_tile(tile_of(tl));
            const int n_start = P.z_is_batch ? zb : n_lo, c_base = P.z_is_batch ? 0 : zb * P.cpg;
            for (int ch = 0; ch < c1 - c0; ++ch) {
                if (!ptx::mbar_wait(raw_empty + rb, pr, abort_flag)) {
                    go = false;
                    break;
                }
                if (A_KMAJOR) { // one [128 rows][32 k] tile per 32 K elements of the stage (columns past K read as zero)
                    ptx::mbar_expect_tx(raw_full + rb, (uint32_t)kAHalfBytes * (KE / 32));
                    for (int h = 0; h < KE / 32; ++h)
                        ptx::tma_load_3d(sRaw + (size_t)rb * P.raw_bytes + (size_t)h * kAHalfBytes, &tmap_x, raw_full + rb,
                                         (c0 + ch) * KE + h * 32, bx * kTileM, zb);
                } else if (P.flat) {
                    ptx::mbar_expect_tx(raw_full + rb, bytes);
                    ptx::tma_load_3d(sRaw + (size_t)rb * P.raw_bytes, &tmap_x, raw_full + rb, 0,
                                     (P.z_is_batch ? c0 + ch : zb * P.nchunks + c0 + ch) * P.flat_rows, n_start); // (whole chunks per group)
                } else {
                    ptx::mbar_expect_tx(raw_full + rb, bytes);
                    ptx::tma_load_5d(sRaw + (size_t)rb * P.raw_bytes, &tmap_x, raw_full + rb, x_start, y_start, z_start,
                                     c_base + (c0 + ch) * P.BC, n_start);
                }
                if (++rb == P.NR) {
                    rb = 0;
                    pr ^= 1u;
                }
            }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (one thread) ----------------
        // 3xTF32 with two MMAs per K=8 step instead of three: the hi and lo filter tiles of a stage are adjacent in shared
        // memory, i.e. one K-major tile of 2*BN rows, so  A_hi x [B_hi ; B_lo]  is ONE MMA of width 2*BN whose result columns
        // [0,BN) are the main accumulator and [BN,2BN) the accumulator of the cross terms; A_lo x B_hi then adds to the
        // latter.  Same tensor-pipe work, a third fewer instructions from the thread that every stage waits for.
        // What this loop does besides its MMAs decides the kernel's rate: the tensor pipe needs 770 / 385 / 240 cycles for the
        // eight MMAs of a stage at BN = 128 / 64 / 32 and queues only two or three instructions, while a wait on a complete
        // mbarrier takes 110-130 cycles, a vote 41, elect 35, a warp barrier 23 — and a taken branch 70 to 250, because the
        // warps of an SM quarter share an instruction cache that the transform warps' unrolled code keeps flushing.  So: one
        // thread, ring positions as running values, the next stage's barriers polled before this stage's MMAs are issued,
        // and a plain stage that is one short straight line; everything rare (waits, group starts) sits outside it.
        // A wait that gives up cuts the loops short (their bounds are running values) and sends the stage's releases to a barrier
        // that nobody waits for, so that the common path has no test for it (one cost it 5 to 12 %).  The releases must not
        // reach the filter slot: with bytes still missing from it, its producer would arrive once more on a phase that expects
        // no further arrival, which is a fault.
        if (ptx::elect_one()) {
            auto idesc_for = [](int n) {
                return REDO ? ptx::idesc_f16(kTileM, n) : (HALF ? ptx::idesc_bf16(kTileM, n) : ptx::idesc_tf32(kTileM, n));
            };
            const uint32_t idesc = idesc_for(P.BN);
            const uint32_t idesc_wide = idesc_for(2 * P.BN);
            // A from TMEM; per instruction K = 8 TF32 values or 16 halves, either way 8 columns of A and 32 bytes of a B row
            auto mma_ts = [](uint32_t d, uint32_t a, uint64_t b, uint32_t id, uint32_t acc) {
                if (HALF)
                    ptx::mma_f16_ts(d, a, b, id, acc);
                else
                    ptx::mma_tf32_ts(d, a, b, id, acc);
            };
            const uint64_t bdesc0 = ptx::smem_desc_k128(ptx::smem_u32(sB));
            const uint32_t b_half16 = b_half >> 4;
            const uint32_t BNu = (uint32_t)P.BN, a_col0 = tmem_base + kACol, NB = (uint32_t)P.NB;
            uint32_t tmem_acc = tmem_base, tmem_small = tmem_base + BNu; // main and cross-term accumulators of the tile
            int tiles_left = items, stages_end = KS, left = 0; // tiles, end of the tile's K stages, stages left in the flush group
            bool ok = true;
            // Ring positions: slot, parity, and what they select.
            uint32_t sa = 0, sb = 0, pa = 0, pb = 0;
            uint64_t bhi = bdesc0;
            uint64_t *release_a = a_empty, *release_b = b_empty;
            auto give_up = [&]() {
                ok = false;
                tiles_left = stages_end = left = 0;
                release_a = trash - sa, release_b = trash - sb;
            };
            bool ready = false, next_ready = false; // the current / the next stage has been seen complete
            auto wait_stage = [&]() {
                if (__builtin_expect(!ready, 0)) {
                    if (!ptx::mbar_wait(a_full + sa, pa, abort_flag) || !ptx::mbar_wait(b_full + sb, pb, abort_flag))
                        give_up();
                }
                ptx::tc_fence_after();
            };
            struct Pos {
                uint32_t sa, sb, pa, pb;
            };
            auto next_pos = [&]() {
                Pos n{sa + 1, sb + 1, pa, pb};
                if (n.sa == (uint32_t)kNA)
                    n.sa = 0, n.pa ^= 1u;
                if (n.sb == NB)
                    n.sb = 0, n.pb ^= 1u;
                return n;
            };
            auto finish_stage = [&](const Pos &n) { // release the stage's slots, go on to the next
                ptx::mma_commit(release_a + sa);
                ptx::mma_commit(release_b + sb);
                sa = n.sa, sb = n.sb, pa = n.pa, pb = n.pb;
                bhi = bdesc0 + (uint64_t)(sb * 2u * b_half16);
                ready = next_ready;
            };
            // One K stage.  The cross terms have their own accumulator: the tensor core truncates (rounds toward zero) its
            // accumulator after every MMA, a bias proportional to the accumulator's magnitude; keeping the small terms away
            // from the big sum removes most of those truncations from it.
            auto plain_stage = [&](uint32_t acc0) {
                wait_stage();
                const Pos n = next_pos();
                // Is the next stage there?  Asked before this stage's MMAs and read after them: the answer travels while they
                // are being issued.
                const bool next_a = ptx::mbar_test_wait(a_full + n.sa, n.pa), next_b = ptx::mbar_test_wait(b_full + n.sb, n.pb);
                const uint32_t ahi_t = a_col0 + sa * 64u, alo_t = ahi_t + 32u;
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    mma_ts(tmem_acc, ahi_t + kk * 8, bhi + 2 * kk, SPLIT ? idesc_wide : idesc, kk == 0 ? acc0 : 1u);
                    if (SPLIT)
                        mma_ts(tmem_small, alo_t + kk * 8, bhi + 2 * kk, idesc, 1u);
                }
                next_ready = next_a && next_b;
                finish_stage(n);
            };
            auto cross_terms = [&](const uint32_t slot_a, const uint64_t hi) { // of one stage: eight MMAs that leave the main accumulator alone
                const uint32_t ahi_t = a_col0 + slot_a * 64u;
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    mma_ts(tmem_small, ahi_t + kk * 8, hi + b_half16 + 2 * kk, idesc, 1u);
                    mma_ts(tmem_small, ahi_t + 32u + kk * 8, hi + 2 * kk, idesc, 1u);
                }
            };
            auto main_terms = [&](uint32_t acc0) {
                const uint32_t ahi_t = a_col0 + sa * 64u;
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)
                    mma_ts(tmem_acc, ahi_t + kk * 8, bhi + 2 * kk, idesc, kk == 0 ? acc0 : 1u);
            };
            uint32_t gpar = 0; // parity of the flush group's drain
            // First stage(s) of a new flush group: the main accumulator restarts from zero, but only after the drain warps have
            // taken the previous group's sum.  The stage's eight cross-term MMAs do not touch the main accumulator and are
            // issued first, so the tensor pipe has work while the drain is in flight; if the stage after it is already there
            // (and belongs to the group), its eight as well.
            auto group_start = [&]() {
                wait_stage();
                if (!ok)
                    return;
                const Pos n = next_pos();
                cross_terms(sa, bhi);
                next_ready = ptx::mbar_test_wait(a_full + n.sa, n.pa) && ptx::mbar_test_wait(b_full + n.sb, n.pb);
                const bool two = next_ready && left >= 2;
                if (two) {
                    ptx::tc_fence_after();
                    cross_terms(n.sa, bdesc0 + (uint64_t)(n.sb * 2u * b_half16));
                }
                if (!ptx::mbar_wait(flushed, gpar, abort_flag)) {
                    give_up();
                    return;
                }
                gpar ^= 1u;
                ptx::tc_fence_after();
                main_terms(0u);
                finish_stage(n);
                --left;
                if (!two)
                    return;
                const Pos n2 = next_pos();
                next_ready = ptx::mbar_test_wait(a_full + n2.sa, n2.pa) && ptx::mbar_test_wait(b_full + n2.sb, n2.pb);
                main_terms(1u);
                finish_stage(n2);
                --left;
            };
            const int FLm = (PP == kNarrow || !SPLIT || P.fl == 0) ? KS : P.fl; // stages per flush group
            for (int tl = 0; tl < tiles_left; ++tl) {
                if (PP) {
                    // before an accumulator region is reused, its previous tile must have been read out
                    const int reg = two_regions ? (tl & 1) : 0, use = two_regions ? (tl >> 1) : tl; // the use-th tile of region reg
                    tmem_acc = tmem_base + (uint32_t)reg * 2u * BNu;
                    tmem_small = tmem_acc + BNu;
                    if (use >= 1) {
                        if (!ptx::mbar_wait(acc_empty + reg, (uint32_t)((use - 1) & 1), abort_flag)) {
                            give_up();
                            break;
                        }
                        ptx::tc_fence_after();
                    }
                }
                for (int g0 = 0; g0 < stages_end; g0 += FLm) {
                    left = min(FLm, KS - g0);
                    if (PP != kNarrow && g0 > 0)
                        group_start();
                    uint32_t acc0 = g0 > 0 ? 1u : 0u;
#pragma unroll 1
                    for (; left > 0; --left, acc0 = 1u)
                        plain_stage(acc0);
                    if (PP != kNarrow && g0 + FLm < stages_end) // (0 after a give-up) fires once every MMA of the group has completed
                        ptx::mma_commit(acc_ready);
                }
                if (ok)
                    ptx::mma_commit((two_regions && (tl & 1)) ? acc_full1 : acc_full);
            }
        }
        __syncwarp();
    } else if (warp >= kSetWarp && warp < kDrainWarp) {
        // ---------------- transform: two sets of four warps taking alternate K stages (and the epilogue of a single tile) --------
        // The per-stage chain  wait -> gather -> tcgen05.st -> wait::st -> arrive  is latency bound (about 750 cycles: 110-130
        // for a wait, 270-310 from the first tcgen05.st to the arrive); two sets halve the time between stages.
        if (!SECOND) {
            if (PP == kWide)
                ptx::reg_dealloc<Regs<PP>::set>();
            else
                ptx::reg_alloc<Regs<PP>::set>();
        }
        const int tset = (warp - kSetWarp) >> 2; // 0 or 1
        const int quarter = warp & 3;            // TMEM lane quarter this warp may access
        const int p = quarter * 32 + lane;       // pixel row inside the tile
        bool alive = true;
        const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16);
        // This set's stages are number tset, tset + 2, ... of the CTA (all tiles in a row): `st` is the next one's index inside
        // the current chunk, `sa` / `pa` its A slot and the parity to wait for (first pass over the ring: every slot is free).
        int st = tset, rb = 0;
        uint32_t sa = (uint32_t)tset, pa = 1u, prw = 0;
        bool valid = false;
        long long y_off = 0;
        // The whole loop is instantiated per kind of gather, so that a stage is short and straight.
        auto transform = [&](auto mode_c, auto rescale_c) {
            constexpr int MODE = decltype(mode_c)::value;
            constexpr bool RESCALE = decltype(rescale_c)::value; // fp16's second pass
            const bool flat = MODE == kGatherFlat || ((MODE == kGatherStride || MODE == kGatherPlain) && P.flat != 0);
            bool raw_ok = true; // this lane has not given up on a raw tile (the warp agrees on it where it asks for an A slot)
            int fetched = 0, frb = 0; // GBMML: chunks asked for, ring slot of the next and the parity that says it is free
            uint32_t fpr = 0;
            const int nfetch = ntl * (c1 - c0);
            for (int tl = 0; tl < items && alive; ++tl) {
                set_tile(tile_of(tl));
                int base_p;
                pixel_geom(p, valid, base_p, y_off);
                float top = 0.f; // fp16: largest magnitude of this thread's operands
                [[maybe_unused]] volatile uint8_t *my_exp = row_exps + (((tl >> twice) & (kExpSlots - 1)) * 2 + tset) * kTileM + p;
                [[maybe_unused]] float factor = 1.f;
                if constexpr (RESCALE) {
                    if (for_sums(tl))
                        factor = row_scale(exponent_of(tl, p));
                }
                if (P.ksplit > 1 && tset == 0)
                    sYoff[p] = valid ? y_off : -1; // read by the split-K reduction, after the cluster barrier
                uint32_t tmask = 0;
                if (MODE < kGatherKMajor && flat && valid) { // which filter taps of this pixel lie inside the (unpadded) input
                    int ul = 0, q = q0 + p;
                    if (P.ipt > 1) {
                        ul = P.by_pw.div(p);
                        q = p - ul * P.Pw;
                    }
                    const int zl = unit0 + ul - P.by_od.div(unit0 + ul) * P.OD, yl = P.by_own.div(q), xl = q - yl * P.own;
                    const int z0 = zl * P.sd - P.pd, y0 = (P.oh0 + yl) * P.sh - P.ph, x0 = (P.ow0 + xl) * P.sw - P.pw;
                    int tap = 0;
                    for (int t = 0; t < P.T3[0]; ++t)
                        for (int r = 0; r < P.T3[1]; ++r)
                            for (int sx = 0; sx < P.T3[2]; ++sx, ++tap) {
                                const int z = z0 + t * P.dil[0], y = y0 + r * P.dil[1], x = x0 + sx * P.dil[2];
                                if (z >= 0 && z < P.xD && y >= 0 && y < P.xH && x >= 0 && x < P.xW)
                                    tmask |= 1u << tap;
                            }
                }
                for (int ch = 0; ch < c1 - c0 && alive; ++ch, st -= P.spc) {
                    if constexpr (MODE == kGatherBand) { // keep NR - 1 chunks in flight
                        for (; fetched < nfetch && fetched < tl * (c1 - c0) + ch + P.NR && alive; ++fetched) {
                            if (fetched >= P.NR) {
                                alive = ptx::mbar_wait_warp(raw_empty + frb, fpr, abort_flag); // (its previous chunk has been read by all)
                            }
                            const int ft = fetched / (c1 - c0), fm = PP ? P.by_ntiles.div((int)blockIdx.x + ft * (int)gridDim.x) : 0;
                            const int fz = PP ? P.by_mtiles.div(fm) : zb, fx = PP ? fm - fz * P.mtiles : bx;
                            band_copy(P, fz, fx * kTileM, ((fx * kTileM - P.band_w) & ~3) + (fetched - ft * (c1 - c0)) * kBandKeys, warp - kSetWarp,
                                      lane, ptx::smem_u32(sRaw + (size_t)frb * P.raw_bytes), raw_full + frb);
                            if (++frb == P.NR) {
                                frb = 0;
                                fpr ^= fetched >= P.NR ? 1u : 0u;
                            }
                        }
                        if (!alive)
                            break;
                    }
                    raw_ok = ptx::mbar_wait(raw_full + rb, prw, abort_flag) && raw_ok; // also by a set without a stage in this chunk
                    const float *raw = reinterpret_cast<const float *>(sRaw + (size_t)rb * P.raw_bytes) + base_p;
                    for (; st < P.spc && alive; st += 2) {
                        const int *ko = sKoff + st * KE;
                        // Is the slot free?  Asked before the gather, read after it.
                        const bool slot_free = ptx::mbar_test_wait(a_empty + sa, pa);
                        // The operands are gathered and split into registers BEFORE the wait for the stage's slot in tensor
                        // memory: when the slot frees, only the two tcgen05.st remain, so a set is one stage ahead in
                        // registers on top of its slots in the ring.  (Announcing a stage only after the next one's gather,
                        // to hide the 200 to 250 cycles of the stores, was 8 % slower: the MMA thread starts later.)
                        // A stage of halves is 64 elements: where they are gathered one by one, two rounds of the same code, 32 each
                        // (see split_words), the slot awaited in the first; row-major rows are 16 reads, whose latencies
                        // in two rounds made a stage 5 % longer (16 x 768 x 3072 on one tile row: 30.0 us, in one round 28.4).
                        constexpr int kRounds = HALF && !A_KMAJOR ? 2 : 1, kParts = (HALF ? 2 : 1) / kRounds;
#pragma unroll 1
                        for (int round = 0; round < kRounds; ++round) {
                        constexpr int kWords = 32 / kRounds; // of hi and of lo in a round
                        uint32_t hi[kWords], lo[kWords];
                        if constexpr (MODE == kGatherBand) {
                            const int i = bx * kTileM + p, k0 = ((bx * kTileM - P.band_w) & ~3) + ((c0 + ch) * kBandStages + st) * kStageK;
                            const int j0 = k0 - i + P.band_w; // band column of the stage's first key
                            const float *brow = reinterpret_cast<const float *>(sRaw + (size_t)rb * P.raw_bytes) + p * kBandPitch + st * kStageK;
                            const int shift = (int)(band_word(P, zb, i, k0) & 3), lo_e = max(-j0, -k0);
                            const int hi_e = i < P.m_rows ? min(2 * P.band_w + 1 - j0, P.m_rows - k0) : 0;
#pragma unroll
                            for (int c = 0; c < 4; ++c) {
                                float v[8];
                                band_take8(brow + 8 * c, shift, lo_e - 8 * c, hi_e - 8 * c, v);
                                split_words<PASSES>(v, hi + 8 * c, lo + 8 * c, top);
                            }
                        } else {
#pragma unroll
                            for (int part = 0; part < kParts; ++part) {
                            const int half = round + part;
                            const int *kh = ko + half * kStageK;
                            const uint8_t *krow = sRaw + (size_t)rb * P.raw_bytes + (size_t)p * 128 + half * kAHalfBytes; // (a stage's second tile follows the first)
                            const float *q = raw; // kGatherPlain: first element of the run
                            int cs = P.cstride;
                            if constexpr (MODE == kGatherPlain) {
                                const int o0 = *kh;
                                const bool off = o0 < 0 || (flat && !((tmask >> (o0 >> 24)) & 1u));
                                q = off ? zero_word : raw + (flat ? (o0 & 0xffffff) : o0);
                                cs = off ? 0 : cs;
                            }
                            constexpr int kGroups = HALF ? 2 : 1; // groups of eight elements that make eight words
#pragma unroll
                            for (int c = 0; c < 4 / kGroups; ++c) {
                                float v[8 * kGroups];
#pragma unroll
                                for (int h = 0; h < kGroups; ++h) {
                                    const int e = kGroups * c + h;
                                    if constexpr (MODE == kGatherPlain) {
#pragma unroll
                                        for (int i = 0; i < 8; ++i)
                                            v[8 * h + i] = q[(8 * e + i) * cs];
                                    } else {
                                        gather8<MODE>(kh + 8 * e, raw, krow, 2 * e, p, tmask, P.cstride, flat, zero_word, v + 8 * h);
                                    }
                                }
                                if constexpr (RESCALE) {
#pragma unroll
                                    for (int i = 0; i < 16; ++i)
                                        v[i] *= factor;
                                }
                                split_words<PASSES>(v, hi + 16 * part + 8 * c, lo + 16 * part + 8 * c, top);
                            }
                            }
                        }
                        if (round == 0) {
                            if (__builtin_expect(!__all_sync(0xffffffffu, slot_free && raw_ok), 0)) {
                                raw_ok = __all_sync(0xffffffffu, raw_ok) != 0;
                                alive = raw_ok && ptx::mbar_wait_warp(a_empty + sa, pa, abort_flag);
                                if (!alive)
                                    break;
                            }
                            ptx::tc_fence_after();
                        }
                        const uint32_t t = t_row + kACol + sa * 64u + round * 16u;
                        if constexpr (kWords == 16) {
                            ptx::tmem_st_32x16(t, hi);
                            ptx::tmem_st_32x16(t + 32u, lo);
                        } else {
                            ptx::tmem_st_32x32(t, hi);
                            if (SPLIT)
                                ptx::tmem_st_32x32(t + 32u, lo);
                        }
                        }
                        if (!alive)
                            break;
                        if (REDO && !(RESCALE && for_sums(tl)))
                            *my_exp = (uint8_t)row_exponent(top);
                        ptx::tmem_st_wait();
                        ptx::tc_fence_before();
                        __syncwarp();
                        if (lane == 0)
                            ptx::mbar_arrive(a_full + sa);
                        sa ^= 2u;
                        pa ^= (sa & 2u) ? 0u : 1u; // back at the set's first slot: the ring's next pass
                    }
                    __syncwarp();
                    if (lane == 0 && alive)
                        ptx::mbar_arrive(raw_empty + rb);
                    if (++rb == P.NR) {
                        rb = 0;
                        prw ^= 1u;
                    }
                }
                if constexpr (RESCALE) {
                    if (!for_sums(tl) && alive) { // the other set's exponents are needed too
                        __syncwarp();
                        if (lane == 0)
                            ptx::mbar_arrive(scanned);
                        alive = ptx::mbar_wait_warp(scanned, (uint32_t)((tl >> 1) & 1), abort_flag);
                    }
                }
            }
        };
        [[maybe_unused]] const uint32_t factor_answer = !PP ? ask_factors() : 0u;
        auto transform_by_mode = [&](auto rescale_c) {
            if constexpr (BAND == 2) {
                transform(std::integral_constant<int, kGatherBand>(), rescale_c);
                ptx::cp_async_wait_all(); // (nothing may be written to the CTA's shared memory after it is gone)
            } else if constexpr (A_KMAJOR) {
                transform(std::integral_constant<int, kGatherKMajor>(), rescale_c);
            } else if (P.cstride && P.BC % kStageK == 0) {
                transform(std::integral_constant<int, kGatherPlain>(), rescale_c);
            } else if (P.cstride) {
                transform(std::integral_constant<int, kGatherStride>(), rescale_c);
            } else if (P.flat) {
                transform(std::integral_constant<int, kGatherFlat>(), rescale_c);
            } else {
                transform(std::integral_constant<int, kGatherTable>(), rescale_c);
            }
        };
        transform_by_mode(second_c);
        if (!PP) {
            // ---------------- epilogue of the only tile ----------------
            // Addresses and store mode first: the MMA thread is still working through the last stages, so this costs nothing.
            // The two sets split the tile's columns.  Code that runs once per CTA comes out of a cold instruction cache, so its
            // length is its cost: small loops.
            const int per_set = P.BN / 2, col0 = tset * per_set, f_tile0 = ntile * P.BN;
            const long long f_glob0 = P.z_is_batch ? 0 : (long long)zb * P.Fg;
            StoreJob J;
            J.y = P.y + f_glob0 * P.ys_f;
            J.bias = P.has_bias ? P.bias + f_glob0 : nullptr;
            J.res = P.res != nullptr ? P.res + f_glob0 * P.ys_f : nullptr;
            J.ys_f = P.ys_f, J.y_off = y_off, J.Fg = P.Fg, J.act = P.act, J.lane = lane, J.valid = valid;
            J.nvalid = __popc(__ballot_sync(0xffffffffu, valid));
            J.y_off0 = __shfl_sync(0xffffffffu, y_off, 0);
            // a 4 KB block per warp: the filter ring is idle once the accumulator is complete (if it is large enough)
            float *stage = reinterpret_cast<float *>(smem + (L.stage_off == L.bar_off ? L.b_off : L.stage_off)) + (warp - kSetWarp) * 1024;
            if (alive)
                alive = ptx::mbar_wait_warp(acc_full, 0u, abort_flag);
            if (SPLIT && P.fl > 0) // the drain warps have written total + last group over the main accumulator
                ptx::named_bar_sync(1, 384);
            [[maybe_unused]] const bool factors = any_factor(factor_answer);
            [[maybe_unused]] float unscale = 1.f;
            if (REDO && alive) {
                const uint32_t e = exponent_of(0, p);
                alive = store_now(e, valid);
                unscale = row_unscale(e);
            }
            if (alive && P.ksplit > 1) {
                // Split-K: column c of the tile is summed by CTA c / cols of the cluster.  Push this CTA's partial sum into that
                // CTA's shared memory, slot [this rank][c % cols][pixel] (consecutive lanes = consecutive words).
                ptx::tc_fence_after();
                const int cols = P.cols, shift = 31 - __clz(cols), me = (int)ptx::cluster_ctarank();
                const uint32_t mine = ptx::smem_u32(sSplit) + (uint32_t)(me * cols * kTileM + p) * 4u;
#pragma unroll 1
                for (int c = col0; c < col0 + per_set; c += 8) {
                    uint32_t v[8], x[8];
                    ptx::tmem_ld_32x8(t_row + (uint32_t)c, v);
                    if (SPLIT)
                        ptx::tmem_ld_32x8(t_row + (uint32_t)(P.BN + c), x);
                    ptx::tmem_ld_wait();
                    float sum[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        sum[j] = join_sums<PASSES>(v[j], SPLIT ? x[j] : 0u);
                    if (REDO && (pass || factors)) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const float filter = factors && f_tile0 + c + j < P.Fg ? __ldg(P.fscale + (long long)zb * P.Fg + f_tile0 + c + j) : 1.f;
                            sum[j] = SECOND ? unscaled(sum[j], factor_halves(unscale), factor_halves(filter)) : sum[j] * filter;
                        }
                    }
                    if (cols >= 8) { // one owner: one address translation; the CTA's own block stays out of the cluster network
                        const int owner = c >> shift;
                        const uint32_t local = mine + (uint32_t)((c & (cols - 1)) * kTileM) * 4u;
                        if (owner == me) {
#pragma unroll
                            for (int j = 0; j < 8; ++j)
                                ptx::st_shared_f32(local + (uint32_t)(j * kTileM) * 4u, sum[j]);
                        } else {
                            const uint32_t remote = ptx::map_to_cta(local, (uint32_t)owner);
#pragma unroll
                            for (int j = 0; j < 8; ++j)
                                ptx::st_dsmem_f32(remote + (uint32_t)(j * kTileM) * 4u, sum[j]);
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const int col = c + j;
                            ptx::st_dsmem_f32(ptx::map_to_cta(mine + (uint32_t)((col & (cols - 1)) * kTileM) * 4u, (uint32_t)(col >> shift)),
                                              sum[j]);
                        }
                    }
                }
            } else if (alive) {
                ptx::tc_fence_after();
                const int blocks = (P.BN / 32 + 1) / 2; // whole 32-column blocks per set
                with_store_mode(store_mode(), J.res != nullptr, P.act, [&](auto mode_c, auto res_c, auto long_c) {
#pragma unroll 1
                for (int c = tset * blocks * 32; c < min(P.BN, (tset + 1) * blocks * 32); c += 32) {
                    float r[32];
#pragma unroll
                    for (int h = 0; h < 32; h += 16) {
                        uint32_t v[16], x[16];
                        ptx::tmem_ld_32x16(t_row + (uint32_t)(c + h), v);
                        if (SPLIT)
                            ptx::tmem_ld_32x16(t_row + (uint32_t)(P.BN + c + h), x);
                        ptx::tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            r[h + j] = join_sums<PASSES>(v[j], SPLIT ? x[j] : 0u);
                    }
                    if (REDO && (pass || factors))
                        unscale_block<SECOND>(r, unscale, P.fscale + (long long)zb * P.Fg, f_tile0 + c, P.Fg, factors, lane);
                    store_block<decltype(mode_c)::value, decltype(res_c)::value, decltype(long_c)::value, 1>(J, r, stage, f_tile0 + c);
                }
                });
            }
        }
    } else if (warp >= kDrainWarp) {
        // ---------------- drain warps: running totals of flushed accumulators; persistent mode: the epilogue ----------------
        if (!SECOND)
            ptx::reg_alloc<Regs<PP>::drain>();
        const int quarter = warp & 3, p = quarter * 32 + lane, FL = SPLIT ? P.fl : 0;
        const int n_groups = FL > 0 ? P.by_fl.div(KS + FL - 1) : 1;
        [[maybe_unused]] const bool factors = PP && any_factor(ask_factors());
        const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16);
        bool alive = true;
        uint32_t gpar = 0; // parity of the next completed group
        if (BAND == 1) {
            for (int tl = 0; tl < ntl && alive; ++tl) {
                set_tile((int)blockIdx.x + tl * (int)gridDim.x);
                alive = ptx::mbar_wait_warp((tl & 1) ? acc_full1 : acc_full, (uint32_t)((tl >> 1) & 1), abort_flag);
                if (!alive)
                    break;
                ptx::tc_fence_after();
                const uint32_t tacc = t_row + (uint32_t)((tl & 1) * 2 * P.BN);
                epilogue_banded<PASSES>(tacc, tacc + (uint32_t)P.BN, 0, P.BN, ntile * P.BN, quarter * 32, bx, zb, P.m_rows, P.band_w, P.y,
                                        reinterpret_cast<float *>(smem + L.stage_off) + quarter * 1024, lane);
                ptx::tc_fence_before();
                __syncwarp();
                if (lane == 0)
                    ptx::mbar_arrive(acc_empty + (tl & 1));
            }
        } else if (PP || FL > 0) {
            float *stage = reinterpret_cast<float *>(smem + L.stage_off) + quarter * 1024;
            auto drain = [&](auto mode_c, auto res_c, [[maybe_unused]] auto long_c) {
            [[maybe_unused]] constexpr int MODE = decltype(mode_c)::value; // (a single tile stores nothing here)
            [[maybe_unused]] constexpr bool RES = decltype(res_c)::value;
            for (int tl = 0; tl < items && alive; ++tl) {
                const int reg = two_regions ? (tl & 1) : 0, use = two_regions ? (tl >> 1) : tl;
                StoreJob J;
                if (PP) { // where the tile goes: worked out while its MMAs run
                    set_tile(tile_of(tl));
                    int base_p;
                    pixel_geom(p, J.valid, base_p, J.y_off);
                    const long long f_glob0 = P.z_is_batch ? 0 : (long long)zb * P.Fg;
                    J.y = P.y + f_glob0 * P.ys_f;
                    J.bias = P.has_bias ? P.bias + f_glob0 : nullptr;
                    J.res = P.res != nullptr ? P.res + f_glob0 * P.ys_f : nullptr;
                    J.ys_f = P.ys_f, J.Fg = P.Fg, J.act = P.act, J.lane = lane;
                    J.nvalid = __popc(__ballot_sync(0xffffffffu, J.valid));
                    J.y_off0 = __shfl_sync(0xffffffffu, J.y_off, 0);
                }
                const uint32_t tmain = t_row + (uint32_t)(reg * 2 * P.BN);
                [[maybe_unused]] const uint32_t tcross = tmain + (uint32_t)P.BN;
                float racc[PP == kNarrow ? 32 : 128]; // the sums of this thread's tile row (narrow: of the block being stored)
                auto take_acc_full = [&]() {
                    alive = ptx::mbar_wait_warp(reg ? acc_full1 : acc_full, PP == kSingle ? 0u : (uint32_t)(use & 1), abort_flag);
                    ptx::tc_fence_after();
                };
                auto release = [&]() { // the MMA thread may start the region's next tile
                    ptx::tc_fence_before();
                    __syncwarp();
                    if (lane == 0)
                        ptx::mbar_arrive(acc_empty + reg);
                };
                [[maybe_unused]] float unscale = 1.f;
                [[maybe_unused]] auto leave_out = [&]() { // fp16, once a tile is complete: not stored in this pass, or not by this item
                    const uint32_t e = exponent_of(tl, p);
                    unscale = row_unscale(e);
                    return !store_now(e, J.valid) || !for_sums(tl);
                };
                if constexpr (PP == kNarrow) {
                    take_acc_full();
                    if (!alive)
                        break;
                    if constexpr (REDO) {
                        if (leave_out()) {
                            release();
                            continue;
                        }
                    }
#pragma unroll 1 // (one copy of the store code: see FastDiv)
                    for (int c = 0; c < P.BN; c += 32) {
#pragma unroll
                        for (int h = 0; h < 32; h += 16) {
                            uint32_t v[16], x[16];
                            ptx::tmem_ld_32x16(tmain + (uint32_t)(c + h), v);
                            if (SPLIT)
                                ptx::tmem_ld_32x16(tcross + (uint32_t)(c + h), x);
                            ptx::tmem_ld_wait();
#pragma unroll
                            for (int j = 0; j < 16; ++j) // hi*hi sum + (lo*hi + hi*lo) sum, one rounded fp32 add
                                racc[h + j] = join_sums<PASSES>(v[j], SPLIT ? x[j] : 0u);
                        }
                        if (c + 32 >= P.BN)
                            release();
                        if (REDO && (pass || factors))
                            unscale_block<SECOND>(racc, unscale, P.fscale + (long long)zb * P.Fg, ntile * P.BN + c, P.Fg, factors, lane);
                        store_block<MODE, RES, decltype(long_c)::value, PP == kNarrow ? 1 : 8>(J, racc, stage, ntile * P.BN + c);
                    }
                } else {
                    // Groups in order, round-to-nearest adds; the MMA thread restarts the main accumulator once a group has been taken.
                    for (int g = 0; g + 1 < n_groups && alive; ++g, gpar ^= 1u) {
                        alive = ptx::mbar_wait_warp(acc_ready, gpar, abort_flag);
                        if (!alive)
                            break;
                        ptx::tc_fence_after();
                        drain_add<PASSES, false>(racc, tmain, 0u, P.BN, g == 0);
                        ptx::tc_fence_before();
                        __syncwarp();
                        if (lane == 0)
                            ptx::mbar_arrive(flushed);
                    }
                    if (alive)
                        take_acc_full();
                    if (!alive)
                        break;
                    if constexpr (PP == kSingle) { // write the total back over the main accumulator for the transform sets' epilogue
                        drain_add<PASSES, false>(racc, tmain, 0u, P.BN, n_groups == 1);
#pragma unroll
                        for (int b = 0; b < 8; ++b)
                            if (b * 16 < P.BN) {
                                uint32_t v[16];
#pragma unroll
                                for (int j = 0; j < 16; ++j)
                                    v[j] = __float_as_uint(racc[b * 16 + j]);
                                ptx::tmem_st_32x16(tmain + (uint32_t)(b * 16), v);
                            }
                        ptx::tmem_st_wait();
                        ptx::tc_fence_before();
                    } else {
                        drain_add<PASSES, SPLIT>(racc, tmain, tcross, P.BN, n_groups == 1);
                        release();
                        if constexpr (REDO) {
                            if (leave_out())
                                continue;
                        }
#pragma unroll 1
                        for (int c = 0; c < P.BN; c += 32) {
                            if (REDO && (pass || factors))
                                unscale_block<SECOND>(racc, unscale, P.fscale + (long long)zb * P.Fg, ntile * P.BN + c, P.Fg, factors, lane);
                            store_block<MODE, RES, decltype(long_c)::value, PP == kNarrow ? 1 : 8>(J, racc, stage, ntile * P.BN + c);
#pragma unroll
                            for (int j = 0; j < 96; ++j) // the next block's sums move down
                                racc[j] = racc[j + 32];
                        }
                    }
                }
            }
            };
            if constexpr (PP == kSingle)
                drain(std::integral_constant<int, kStoreAny>(), std::integral_constant<bool, false>(), std::integral_constant<bool, false>()); // (stores nothing)
            else
                with_store_mode(store_mode(), P.res != nullptr, P.act, drain);
            if (!PP && FL > 0) // (also after a wait gave up: the transform sets wait here)
                ptx::named_bar_sync(1, 384);
        }
    }
}
// The rare second pass as a call, with the registers the block was launched with: as a second inlined copy it cost every launch
// about 0.3 us and a few per cent of the persistent kernels' rate (more spilled registers), as a loop around the first far more.
template <bool A_KMAJOR, int PASSES, int PP>
__device__ __noinline__ void igemm_second_pass(const CUtensorMap *tmap_x, const CUtensorMap *tmap_bhi, const CUtensorMap *tmap_blo, const IgemmParams *P,
                                               uint8_t *smem, uint32_t tmem_base) {
    igemm_pass<A_KMAJOR, PASSES, PP, 0, true>(*tmap_x, *tmap_bhi, *tmap_blo, *P, CtaSmem(smem, *P), tmem_base, CtaPlace(PP, *P));
}

template <bool A_KMAJOR, int PASSES, int PP = kSingle, int BAND = 0>
__global__ void __launch_bounds__(kThreads, 1)
k_igemm(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_bhi,
        const __grid_constant__ CUtensorMap tmap_blo, const __grid_constant__ IgemmParams P) {
    constexpr bool LINK = PP == kSingle && BAND == 0; // may be part of a chain of launches
    constexpr bool REDO = PASSES == kMathF16x3;
    constexpr int KE = PASSES == kMathBf16x3 || PASSES == kMathF16x3 ? 64 : 32;
    extern __shared__ uint8_t smem_raw[];
    // 1024-byte alignment for the swizzled operand tiles
    uint8_t *smem = smem_raw + ((1024u - (ptx::smem_u32(smem_raw) & 1023u)) & 1023u);
    const CtaSmem S(smem, P);
    const CtaPlace at(PP, P);
    const int warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        init_barriers(S.bars, BAND == 2 ? 256 : 1); // (GBMML: every transform thread)
        *S.abort_flag = 0;
        *S.zero_word = 0.f;
        *S.left_over = 0;
        ptx::fence_mbar_init();
        ptx::prefetch_tmap(&tmap_x);
        ptx::prefetch_tmap(&tmap_bhi);
        ptx::prefetch_tmap(&tmap_blo);
    }
    for (int i = threadIdx.x; i < P.spc * KE; i += kThreads)
        S.sKoff[i] = P.koff[i];
    if (warp == 2) {
        ptx::tmem_alloc(S.tmem_slot, kTmemCols);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem_base = *S.tmem_slot;
    // Everything above touched only this CTA's own state and the plan's constant table, so under programmatic dependent
    // launch it overlaps the tail of the preceding kernel; from here on the kernel reads what that kernel wrote.
    // In a chain of launches that do not need one another's results (see `link`) the first lets its successor start only once
    // the kernel before the chain has completed, and the others do not wait at all.
    if (LINK && P.link == kLinkFirst) {
        ptx::grid_dep_wait();
        ptx::grid_dep_launch_dependents();
    } else {
        ptx::grid_dep_launch_dependents();
        if (!LINK || P.link != kLinkNext)
            ptx::grid_dep_wait();
    }


    igemm_pass<A_KMAJOR, PASSES, PP, BAND, false>(tmap_x, tmap_bhi, tmap_blo, P, S, tmem_base, at);
    if constexpr (REDO) {
        ptx::tc_fence_before();
        __syncthreads();
        if (__builtin_expect(*S.left_over != 0 && *S.abort_flag == 0, 0)) {
            // Nothing of the first pass is in flight: its barriers are left behind for a fresh set.
            if (threadIdx.x == 0) {
                init_barriers(S.bars + kBarBytes / 8, 1);
                ptx::fence_mbar_init();
            }
            ptx::fence_proxy_async_smem(); // the filter ring may have held blocks of a tile being stored
            __syncthreads();
            ptx::tc_fence_after();
            if (warp < kSetWarp || (warp < kDrainWarp && PP == kWide)) // back to what the block was launched with: 128 a thread
                ptx::reg_alloc<128>();
            else
                ptx::reg_dealloc<128>();
            igemm_second_pass<A_KMAJOR, PASSES, PP>(&tmap_x, &tmap_bhi, &tmap_blo, &P, smem, tmem_base);
        }
    }

    // ---------------- split-K: reduction across the cluster ----------------
    // Every thread of every CTA of the cluster reaches the barrier (all waits above are bounded).
    if (!PP && P.ksplit > 1) {
        const int ntile = at.ntile, zb = at.zb;
        if (warp >= kSetWarp && warp < kSetWarp + 4) {
            // The bias / residual values the reduction below adds start their way to L1 while the cluster meets.  Set 0's
            // threads do it, for the row each of them wrote into sYoff itself (both halves of the CTA's column slice).
            const int et = threadIdx.x - kSetWarp * 32, cols = P.cols;
            const long long y_off = S.sYoff[et];
            const int f = ntile * P.BN + (int)ptx::cluster_ctarank() * cols;
            const long long f_glob0 = P.z_is_batch ? 0 : (long long)zb * P.Fg;
            if (y_off >= 0 && P.ys_f == 1) {
                if (P.res != nullptr)
                    for (int i = 0; i < cols && f + i < P.Fg; i += 8)
                        ptx::prefetch_l1(P.res + y_off + f_glob0 + f + i);
                if (P.has_bias && et == 0)
                    for (int i = 0; i < cols && f + i < P.Fg; i += 8)
                        ptx::prefetch_l1(P.bias + f_glob0 + f + i);
            }
        }
        ptx::cluster_sync_all(); // every CTA's pushes have landed; nothing touches a peer's memory after this
        if (warp >= kSetWarp && warp < kDrainWarp) {
            const int et = threadIdx.x - kSetWarp * 32;
            const long long y_off = S.sYoff[et & (kTileM - 1)];
            if (y_off >= 0 && *S.abort_flag == 0) {
                const long long f_glob0 = P.z_is_batch ? 0 : (long long)zb * P.Fg;
                float *yp = P.y + y_off + f_glob0 * P.ys_f;
                const float *bp = P.has_bias ? P.bias + f_glob0 : nullptr;
                const float *rp = P.res != nullptr ? P.res + y_off + f_glob0 * P.ys_f : nullptr;
                const int rank = (int)ptx::cluster_ctarank();
                // 16-byte stores need filters contiguous in y, 16-byte aligned rows, and column runs of at least 2
                const bool red_vec = (P.ys_f == 1) && ((P.ys_p & 3) == 0) && ((P.ys_n & 3) == 0) && ((P.Fg & 3) == 0) &&
                                     ((reinterpret_cast<uintptr_t>(P.y) & 15) == 0) && (P.cols >= 4) &&
                                     (P.res == nullptr || (reinterpret_cast<uintptr_t>(P.res) & 15) == 0);
#define PETB200_RED(ACT_) \
    cluster_reduce_store<ACT_>(S.sSplit, P.ksplit, rank, P.cols, et, ntile * P.BN, P.Fg, bp, rp, yp, P.ys_f, red_vec)
                switch (P.act) {
                case PETB200_ACT_RELU: PETB200_RED(PETB200_ACT_RELU); break;
                case PETB200_ACT_SIGMOID: PETB200_RED(PETB200_ACT_SIGMOID); break;
                case PETB200_ACT_TANH: PETB200_RED(PETB200_ACT_TANH); break;
                case PETB200_ACT_GELU: PETB200_RED(PETB200_ACT_GELU); break;
                default: PETB200_RED(PETB200_ACT_NONE); break;
                }
#undef PETB200_RED
            }
        }
    }

    // ---------------- teardown ----------------
    if (*S.abort_flag) {
        // give copies that may still be in flight time to land before the CTA's shared memory is released
        uint64_t t0 = ptx::globaltimer_ns();
        while (ptx::globaltimer_ns() - t0 < 200000ull)
            __nanosleep(1000);
        if (threadIdx.x == 0 && P.status)
            atomicExch(P.status, 1);
    }
    ptx::tc_fence_before();
    __syncthreads();
    if (warp == 2)
        ptx::tmem_dealloc(tmem_base, kTmemCols);
    if (LINK && P.link == kLinkNext) // whoever waits for this launch waits for the ones before it in the chain too
        ptx::grid_dep_wait();
}

typedef void (*KernelFn)(CUtensorMap, CUtensorMap, CUtensorMap, IgemmParams);
// The kernel for one arithmetic, in a file each (they are what takes long to compile): igemm_tf32.cu, igemm_f16.cu, igemm_opt.cu (one
// TF32 product, bf16), igemm_band.cu.  The bound of its waits is a variable of the file's device code.
typedef int (*SetWaitLimitFn)(unsigned long long);
KernelFn igemm_tf32x3(bool a_kmajor, int pp);
KernelFn igemm_f16x3(bool a_kmajor, int pp);
KernelFn igemm_tf32x1(bool a_kmajor, int pp);
KernelFn igemm_bf16x3(bool a_kmajor, int pp);
KernelFn igemm_band(int band, int pp); // 1: G2BMM (kNarrow only), 2: GBMML
int igemm_tf32_wait_limit(unsigned long long ns);
int igemm_f16_wait_limit(unsigned long long ns);
int igemm_opt_wait_limit(unsigned long long ns);
int igemm_band_wait_limit(unsigned long long ns);
#define PETB200_IGEMM_PICK(NAME, MATH)                                                                                            \
    KernelFn NAME(bool a_kmajor, int pp) {                                                                                          \
        if (a_kmajor)                                                                                                               \
            return pp == kSingle ? k_igemm<true, MATH> : (pp == kNarrow ? k_igemm<true, MATH, kNarrow> : k_igemm<true, MATH, kWide>);    \
        return pp == kSingle ? k_igemm<false, MATH> : (pp == kNarrow ? k_igemm<false, MATH, kNarrow> : k_igemm<false, MATH, kWide>);    \
    }
#define PETB200_IGEMM_WAIT_LIMIT(NAME)                                                                                            \
    int NAME(unsigned long long ns) {                                                                                               \
        return cudaMemcpyToSymbol(ptx::g_mbar_wait_limit_ns, &ns, sizeof ns) == cudaSuccess ? PETB200_OK : PETB200_ERR_CUDA;          \
    }

} // namespace petb200
