// Implicit-GEMM convolution / matmul on the 5th-generation tensor cores (tcgen05) with error-compensated TF32.
//
//   D[pixel, filter] = sum_k A[pixel, k] * B[filter, k]            k = (channel chunk, tap, channel in chunk)
//
// A tile is 128 pixels x BN filters (BN = 32, 64 or 128); a CTA computes one, or several in turn (persistent tiles).  The fp32
// accumulators and the A operand live in tensor memory (TMEM).  Sixteen warps:
//   0      TMA producer for the packed weights: per K stage (32 words of K) one 2-D tile of B_hi and one of B_lo, straight into
//          128-byte-swizzled K-major shared memory.
//   1      one thread issues, per K=8 step, the three products of 3xTF32 as two MMAs — A_hi x [B_hi;B_lo] (one MMA of width
//          2*BN: the hi*hi sum and the hi*lo sum in adjacent accumulators) and A_lo x B_hi — and commits the stage release
//          barriers.
//   2      TMA producer for the RAW activation tile of one channel chunk (all taps share it): a 5-D box
//          [images, channels, depth, rows, cols] of the NC(D)HW input, zero-filled outside the tensor, which is exactly the
//          convolution's zero padding.  Box start along W is rounded down to 16 bytes.  (3 is idle.)
//   4-7, 8-11  two transform sets taking alternate K stages.  Thread p owns pixel p of the tile: for every K stage it gathers its
//          32 values from the raw tile (fixed strides where the channel chunk allows, else through a precomputed offset table:
//          tap shift, dilation, channel plane), splits each fp32 into hi (top 19 bits) and lo = x - hi, and writes both to
//          TMEM with tcgen05.st, which leaves the shared-memory read port to B alone.  With one tile per CTA they also store it.
//   12-15  drain warps.  The tensor core truncates its fp32 accumulator after every MMA, so long K ranges empty the main
//          accumulator every few stages into a running total that these warps hold.  With persistent tiles they store a finished
//          tile (tcgen05.ld -> +bias -> activation -> global stores in the way the layout of y allows, see store_block) while
//          the transform sets run on into the next.
//
// Variants (template parameters): 3xTF32 (default), one TF32 pass, error-compensated bf16 (64 K elements per stage, K = 16 per
// MMA); one tile per CTA or persistent tiles; the banded products.
// Split-K: the ksplit CTAs of one output tile form a thread-block cluster and exchange their partial sums through
// distributed shared memory (pushes into the owner's landing area, one cluster barrier, reduction in rank order).
// Every wait on an mbarrier is bounded (~2 s) and reports through a status word instead of hanging the GPU.
// TMA loads are per CTA (no cluster-wide loads of any kind).
#include "common.h"
#include "tc_ptx.cuh"
#include <algorithm>
#include <array>
#include <cstdlib>
#include <map>
#include <type_traits>

namespace petb200 {

constexpr int kTileM = 128;
constexpr int kStageK = 32;               // 32-bit words per K stage = one 128-byte swizzle row (32 TF32 values or 64 bf16)
// values of the kernel's PASSES parameter: error-compensated TF32 (three products per multiply), one TF32 product, and
// error-compensated bf16 (hi/lo bf16 halves, three products, K = 16 per instruction: half the MMAs of 3xTF32 per K)
constexpr int kMathTf32x3 = 3, kMathTf32x1 = 1, kMathBf16x3 = 16;
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
// The compiler sees one limit for all roles (128 a thread) and spills in the persistent instantiations: 3xTF32 wide 76 bytes
// stored / 176 loaded (convolutions), 64 / 152 (matmul), narrow 68 / 100 and 56 / 76, banded 20 / 28 .. 60 / 144, bf16 up to
// 140 / 328; single-tile instantiations none.
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

// Launches in one stream that write disjoint parts of y and read only what was written before the first of them run side by side
// under programmatic dependent launch (without it they run one after the other, which gives the same).
enum { kLinkNone = 0, kLinkFirst = 1, kLinkNext = 2 };
struct IgemmParams {
    int link;               // position in such a chain
    FastDiv by_ntiles, by_mtiles, by_tpi, by_pw, by_od, by_own, by_ohn, by_row_tiles; // (made by set_divisors)
    int Pw, units;          // pixels of one output plane (one image, one depth slice); number of such planes
    int OD, OH, OW;         // full output extents (for addressing y)
    int ohn, own, oh0, ow0; // output window actually computed (ohn*own = Pw)
    int sd, sh, sw, pd, ph, pw;
    int x0;                 // box origin along W (multiple of 4, may be negative)
    int RN, RD, RH, RW, BC; // raw box extents
    int nchunks, spc;       // channel chunks; K stages per chunk
    int ke;                 // K elements per stage: 32 (TF32) or 64 (bf16, two per 32-bit word)
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
    int T3[3], dil[3];      // filter extents and dilations (flat only: for the tap mask)
    int xD, xH, xW;         // input extents (flat only)
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
};

struct SmemLayout {
    uint32_t b_off, raw_off, koff_off, split_off, stage_off, bar_off, total;
};
__host__ __device__ inline SmemLayout smem_layout(const IgemmParams &P) {
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
    L.total = L.bar_off + 384;
    return L;
}

static void set_divisors(IgemmParams &P) {
    P.by_ntiles.set(P.ntiles), P.by_mtiles.set(P.mtiles), P.by_tpi.set(P.tpi), P.by_pw.set(P.Pw);
    P.by_od.set(P.OD), P.by_own.set(P.own), P.by_ohn.set(P.ohn), P.by_row_tiles.set(P.row_tiles);
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

// Operands of one tile row, eight 32-bit words at a time (a K stage is four such pieces: 32 TF32 values, or 64 bf16 in pairs),
// split into hi/lo parts — TF32: hi = top 19 bits, lo = x - hi, one value per word; bf16: hi = bf16(x), lo = bf16(x - hi), two
// values per word, the lower K index in the low half; a single pass rounds instead.
// (A stage is 200 to 300 instructions that every transform warp fetches again for every stage — the SM quarter's first-level
// instruction cache does not hold them — at about five cycles each, which is what bounds narrow tiles.  As a rolled loop of
// eight elements it was no faster: the branches and the shorter runs of independent loads cost what the fetches did.)
template <int PASSES> __device__ __forceinline__ void split_words(const float *v, uint32_t *hi, uint32_t *lo) {
    if (PASSES == kMathBf16x3) {
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
__device__ __forceinline__ void cluster_reduce_store(const float *stage, int ksplit, int rank, int BN, int et /*0..255*/,
                                                     int f_tile0, int Fg, const float *bias, const float *rp, float *yp /*this pixel, filter 0*/,
                                                     long long ys_f, bool vec_ok) {
    const int cols = BN / ksplit, px = et & (kTileM - 1), half = et >> 7;
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
template <bool CROSS>
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
                racc[b * 16 + j] = CROSS ? x + __uint_as_float(c[j]) : x;
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
template <bool RES>
__device__ __forceinline__ void store_any(const StoreJob &J, const float *bias, const float *r, int f0) {
    const int nf = J.valid ? J.Fg - f0 : 0; // filters of this thread's row
    const bool relu = J.act == PETB200_ACT_RELU;
    const float bv = bias != nullptr && f0 + J.lane < J.Fg ? __ldg(bias + f0 + J.lane) : 0.f; // lane j holds filter j's
    float *dst = J.y + J.y_off + (long long)f0 * J.ys_f;
    const float *rs = RES ? J.res + J.y_off + (long long)f0 * J.ys_f : nullptr;
#pragma unroll
    for (int j = 0; j < 32; ++j, dst += J.ys_f) {
        float v = r[j] + __shfl_sync(0xffffffffu, bv, j);
        if (RES)
            v += j < nf ? __ldg(rs + (long long)j * J.ys_f) : 0.f;
        if (j < nf)
            *dst = relu ? fmaxf(v, 0.f) : v;
    }
}
// This thread's row through one of the long activations, four filters at a time, with bias and residual.
__device__ __forceinline__ void activate_block(const StoreJob &J, float *r, float *stage, int f0) {
    const int lane = J.lane;
#pragma unroll
    for (int j = 0; j < 32; ++j)
        stage[j * 32 + lane] = r[j];
    const float *rp = J.res != nullptr && J.valid ? J.res + J.y_off + (long long)f0 * J.ys_f : nullptr;
#pragma unroll 1
    for (int j = 0; j < 32 && f0 + j < J.Fg; j += 4) {
        float v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            v[i] = stage[(j + i) * 32 + lane];
            if (f0 + j + i < J.Fg) {
                if (J.bias != nullptr)
                    v[i] += __ldg(J.bias + f0 + j + i);
                if (rp != nullptr)
                    v[i] += __ldg(rp + (long long)(j + i) * J.ys_f);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
            stage[(j + i) * 32 + lane] = apply_act(v[i], J.act);
    }
#pragma unroll
    for (int j = 0; j < 32; ++j)
        r[j] = stage[j * 32 + lane];
    __syncwarp();
}
template <int MODE, bool RES>
__device__ __forceinline__ void store_block(const StoreJob &J, float *r /*32 sums*/, float *stage, int f0) {
    const int lane = J.lane;
    __syncwarp(); // the previous block has been read
    const float *bias = J.bias;
    if (__builtin_expect(J.act > PETB200_ACT_RELU, 0)) {
        activate_block(J, r, stage, f0);
        bias = nullptr;
        if (RES) { // the residual has been added
            StoreJob R = J;
            R.bias = R.res = nullptr, R.act = PETB200_ACT_NONE;
            store_block<MODE, false>(R, r, stage, f0);
            return;
        }
    }
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
        store_any<RES>(J, bias, r, f0);
    }
}
// f(mode, with residual) as compile-time constants: the loops around store_block are instantiated per way of storing.
template <typename F> __device__ __forceinline__ void with_store_mode(int mode, bool res, F &&f) {
    const std::integral_constant<bool, true> yes;
    const std::integral_constant<bool, false> no;
    if (mode == kStorePixels)
        res ? f(std::integral_constant<int, kStorePixels>(), yes) : f(std::integral_constant<int, kStorePixels>(), no);
    else if (mode == kStoreFilters)
        res ? f(std::integral_constant<int, kStoreFilters>(), yes) : f(std::integral_constant<int, kStoreFilters>(), no);
    else if (mode == kStoreRows)
        res ? f(std::integral_constant<int, kStoreRows>(), yes) : f(std::integral_constant<int, kStoreRows>(), no);
    else
        res ? f(std::integral_constant<int, kStoreAny>(), yes) : f(std::integral_constant<int, kStoreAny>(), no);
}

// BAND: 0 ordinary operands; 1 G2BMM (banded epilogue, key windows per tile; persistent row-major mode only); 2 GBMML (A operand
// gathered from the band in global memory; row-major mode only).  Kernels of their own, so that the others carry none of it.
template <bool A_KMAJOR, int PASSES, int PP = kSingle, int BAND = 0>
__global__ void __launch_bounds__(kThreads, 1)
k_igemm(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_bhi,
        const __grid_constant__ CUtensorMap tmap_blo, const IgemmParams P) {
    constexpr bool LINK = PP == kSingle && BAND == 0; // may be part of a chain of launches
    extern __shared__ uint8_t smem_raw[];
    // 1024-byte alignment for the swizzled operand tiles
    uint8_t *smem = smem_raw + ((1024u - (ptx::smem_u32(smem_raw) & 1023u)) & 1023u);
    const SmemLayout L = smem_layout(P);
    uint8_t *sB = smem + L.b_off;
    uint8_t *sRaw = smem + L.raw_off;
    int *sKoff = reinterpret_cast<int *>(smem + L.koff_off);
    float *sSplit = reinterpret_cast<float *>(smem + L.split_off);
    long long *sYoff = reinterpret_cast<long long *>(smem + L.split_off + 512u * (uint32_t)P.BN); // split-K only
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + L.bar_off);
    // barrier slots
    uint64_t *raw_full = bars, *raw_empty = bars + kMaxNR;
    uint64_t *b_full = bars + 2 * kMaxNR, *b_empty = b_full + kMaxNB; // up to kMaxNB stages
    uint64_t *a_full = b_empty + kMaxNB, *a_empty = a_full + 4;       // up to 4 stages
    uint64_t *acc_full = a_empty + 4;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_full + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(acc_full + 2);
    float *zero_word = reinterpret_cast<float *>(acc_full + 3); // holds 0.0f: what a masked-off filter tap reads
    uint64_t *acc_ready = acc_full + 4; // a group of `fl` K stages has been accumulated: the main accumulator may be drained
    uint64_t *flushed = acc_full + 5;   // the four drain warps have drained it: the MMA warp may restart it
    uint64_t *acc_full1 = acc_full + 6; // persistent mode: the second accumulator region is complete
    uint64_t *trash = acc_full + 9;     // takes the MMA thread's releases after it gave up
    uint64_t *acc_empty = acc_full + 7; // [2]: the drain warps have read accumulator region 0 / 1 out

    constexpr bool SPLIT = PASSES != kMathTf32x1; // hi/lo operands, two accumulators
    constexpr bool BF = PASSES == kMathBf16x3;
    constexpr int KE = BF ? 64 : 32;              // K elements per stage
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int ntile = PP ? 0 : (int)blockIdx.y / P.ksplit; // (persistent mode: set per tile by set_tile)
    const int ksp = PP ? 0 : (int)blockIdx.y - ntile * P.ksplit;
    int zb = PP ? 0 : (int)blockIdx.z;
    const uint32_t b_half = (uint32_t)P.BN * 128u;
    // TMEM columns: [0,BN) accumulator of the hi*hi products, [BN,2*BN) accumulator of the two small cross terms (persistent
    // narrow tiles: a second such pair behind them), [256,512) the A stages
    constexpr uint32_t kTmemCols = 512, kACol = 256;
    constexpr bool two_regions = PP == kNarrow;

    if (threadIdx.x == 0) {
        for (int i = 0; i < kMaxNR; ++i) {
            ptx::mbar_init(raw_full + i, BAND == 2 ? 256 : 1); // (GBMML: every transform thread)
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
        ptx::mbar_init(acc_ready, 1);
        ptx::mbar_init(flushed, 4);
        ptx::mbar_init(acc_full1, 1);
        ptx::mbar_init(trash, 1);
        ptx::mbar_init(acc_empty, 4);
        ptx::mbar_init(acc_empty + 1, 4);
        *abort_flag = 0;
        *zero_word = 0.f;
        ptx::fence_mbar_init();
        ptx::prefetch_tmap(&tmap_x);
        ptx::prefetch_tmap(&tmap_bhi);
        ptx::prefetch_tmap(&tmap_blo);
    }
    for (int i = threadIdx.x; i < P.spc * KE; i += kThreads)
        sKoff[i] = P.koff[i];
    if (warp == 2) {
        ptx::tmem_alloc(tmem_slot, kTmemCols);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
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

    // Tile origin in the input: first image, depth slice, row and (16-byte aligned) column of the raw box.  `bx` is the
    // pixel-tile index: blockIdx.x, or in persistent mode every gridDim.x-th tile from there.
    int bx = (int)blockIdx.x;
    const int ntl = PP ? (P.tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 1; // tiles of this CTA
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
    // split-K: this CTA reduces the channel chunks [c0, c1)
    const int c0 = (int)((long long)ksp * P.nchunks / P.ksplit), c1 = (int)((long long)(ksp + 1) * P.nchunks / P.ksplit);
    const int KS = (c1 - c0) * P.spc;

    if (warp < kSetWarp)
        ptx::reg_dealloc<Regs<PP>::control>();
    if (warp == 0) {
        // ---------------- packed-weight producer (one thread) ----------------
        if (lane == 0) {
            int sb = 0;
            uint32_t pb = 1; // first pass over the ring: every slot is free
            bool go = true;
            for (int tl = 0; tl < ntl && go; ++tl) {
                if (PP)
                    set_tile((int)blockIdx.x + tl * (int)gridDim.x);
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
            for (int tl = 0; tl < ntl && go; ++tl) {
            if (tl > 0)
                set_tile((int)blockIdx.x + tl * (int)gridDim.x);
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
                                     ((c_base + (c0 + ch) * P.BC) / P.BC) * P.flat_rows, n_start);
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
            const uint32_t idesc = BF ? ptx::idesc_bf16(kTileM, P.BN) : ptx::idesc_tf32(kTileM, P.BN);
            const uint32_t idesc_wide = BF ? ptx::idesc_bf16(kTileM, 2 * P.BN) : ptx::idesc_tf32(kTileM, 2 * P.BN);
            // A from TMEM; per instruction K = 8 TF32 values or 16 bf16 values, either way 8 columns of A and 32 bytes of a B row
            auto mma_ts = [](uint32_t d, uint32_t a, uint64_t b, uint32_t id, uint32_t acc) {
                if (BF)
                    ptx::mma_bf16_ts(d, a, b, id, acc);
                else
                    ptx::mma_tf32_ts(d, a, b, id, acc);
            };
            const uint64_t bdesc0 = ptx::smem_desc_k128(ptx::smem_u32(sB));
            const uint32_t b_half16 = b_half >> 4;
            const uint32_t BNu = (uint32_t)P.BN, a_col0 = tmem_base + kACol, NB = (uint32_t)P.NB;
            uint32_t tmem_acc = tmem_base, tmem_small = tmem_base + BNu; // main and cross-term accumulators of the tile
            int tiles_left = ntl, stages_end = KS, left = 0; // tiles, end of the tile's K stages, stages left in the flush group
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
        if (PP == kWide)
            ptx::reg_dealloc<Regs<PP>::set>();
        else
            ptx::reg_alloc<Regs<PP>::set>();
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
        auto transform = [&](auto mode_c) {
            constexpr int MODE = decltype(mode_c)::value;
            const bool flat = MODE == kGatherFlat || ((MODE == kGatherStride || MODE == kGatherPlain) && P.flat != 0);
            bool raw_ok = true; // this lane has not given up on a raw tile (the warp agrees on it where it asks for an A slot)
            int fetched = 0, frb = 0; // GBMML: chunks asked for, ring slot of the next and the parity that says it is free
            uint32_t fpr = 0;
            const int nfetch = ntl * (c1 - c0);
            for (int tl = 0; tl < ntl && alive; ++tl) {
                set_tile((int)blockIdx.x + tl * (int)gridDim.x);
                int base_p;
                pixel_geom(p, valid, base_p, y_off);
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
                        uint32_t hi[32], lo[32];
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
                                split_words<PASSES>(v, hi + 8 * c, lo + 8 * c);
                            }
                        } else {
                            const uint8_t *krow = sRaw + (size_t)rb * P.raw_bytes + (size_t)p * 128;
                            const float *q = raw; // kGatherPlain: first element of the run
                            int cs = P.cstride;
                            if constexpr (MODE == kGatherPlain) {
                                const int o0 = *ko;
                                const bool off = o0 < 0 || (flat && !((tmask >> (o0 >> 24)) & 1u));
                                q = off ? zero_word : raw + (flat ? (o0 & 0xffffff) : o0);
                                cs = off ? 0 : cs;
                            }
#pragma unroll
                            for (int c = 0; c < 4; ++c) {
                                float v[BF ? 16 : 8];
#pragma unroll
                                for (int h = 0; h < (BF ? 2 : 1); ++h) { // (bf16: the second tile of a row-major stage follows the first)
                                    const int e = BF ? 2 * c + h : c;     // group of eight K elements
                                    if constexpr (MODE == kGatherPlain) {
                                        if (BF && e == 4) { // (64 elements: two runs of 32)
                                            const int o0 = ko[32];
                                            const bool off = o0 < 0 || (flat && !((tmask >> (o0 >> 24)) & 1u));
                                            q = off ? zero_word : raw + (flat ? (o0 & 0xffffff) : o0);
                                            cs = off ? 0 : P.cstride;
                                        }
#pragma unroll
                                        for (int i = 0; i < 8; ++i)
                                            v[8 * h + i] = q[(8 * (BF ? e & 3 : e) + i) * cs];
                                    } else {
                                        gather8<MODE>(ko + 8 * e, raw, krow + (e >> 2) * kAHalfBytes, 2 * (e & 3), p, tmask, P.cstride, flat, zero_word, v + 8 * h);
                                    }
                                }
                                split_words<PASSES>(v, hi + 8 * c, lo + 8 * c);
                            }
                        }
                        if (__builtin_expect(!__all_sync(0xffffffffu, slot_free && raw_ok), 0)) {
                            raw_ok = __all_sync(0xffffffffu, raw_ok) != 0;
                            alive = raw_ok && ptx::mbar_wait_warp(a_empty + sa, pa, abort_flag);
                            if (!alive)
                                break;
                        }
                        ptx::tc_fence_after();
                        const uint32_t t = t_row + kACol + sa * 64u;
                        ptx::tmem_st_32x32(t, hi);
                        if (SPLIT)
                            ptx::tmem_st_32x32(t + 32u, lo);
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
            }
        };
        if constexpr (BAND == 2) {
            transform(std::integral_constant<int, kGatherBand>());
            ptx::cp_async_wait_all(); // (nothing may be written to the CTA's shared memory after it is gone)
        } else if constexpr (A_KMAJOR) {
            transform(std::integral_constant<int, kGatherKMajor>());
        } else if (P.cstride && P.BC % kStageK == 0) {
            transform(std::integral_constant<int, kGatherPlain>());
        } else if (P.cstride) {
            transform(std::integral_constant<int, kGatherStride>());
        } else if (P.flat) {
            transform(std::integral_constant<int, kGatherFlat>());
        } else {
            transform(std::integral_constant<int, kGatherTable>());
        }
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
            if (alive && P.ksplit > 1) {
                // Split-K: column c of the tile is summed by CTA c / cols of the cluster.  Push this CTA's partial sum into that
                // CTA's shared memory, slot [this rank][c % cols][pixel] (consecutive lanes = consecutive words).
                ptx::tc_fence_after();
                const int cols = P.BN / P.ksplit, shift = 31 - __clz(cols), me = (int)ptx::cluster_ctarank();
                const uint32_t mine = ptx::smem_u32(sSplit) + (uint32_t)(me * cols * kTileM + p) * 4u;
#pragma unroll 1
                for (int c = col0; c < col0 + per_set; c += 8) {
                    uint32_t v[8], x[8];
                    ptx::tmem_ld_32x8(t_row + (uint32_t)c, v);
                    if (SPLIT)
                        ptx::tmem_ld_32x8(t_row + (uint32_t)(P.BN + c), x);
                    ptx::tmem_ld_wait();
                    if (cols >= 8) { // one owner: one address translation; the CTA's own block stays out of the cluster network
                        const int owner = c >> shift;
                        const uint32_t local = mine + (uint32_t)((c & (cols - 1)) * kTileM) * 4u;
                        if (owner == me) {
#pragma unroll
                            for (int j = 0; j < 8; ++j)
                                ptx::st_shared_f32(local + (uint32_t)(j * kTileM) * 4u, SPLIT ? __uint_as_float(v[j]) + __uint_as_float(x[j]) : __uint_as_float(v[j]));
                        } else {
                            const uint32_t remote = ptx::map_to_cta(local, (uint32_t)owner);
#pragma unroll
                            for (int j = 0; j < 8; ++j)
                                ptx::st_dsmem_f32(remote + (uint32_t)(j * kTileM) * 4u, SPLIT ? __uint_as_float(v[j]) + __uint_as_float(x[j]) : __uint_as_float(v[j]));
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const int col = c + j;
                            ptx::st_dsmem_f32(ptx::map_to_cta(mine + (uint32_t)((col & (cols - 1)) * kTileM) * 4u, (uint32_t)(col >> shift)),
                                              SPLIT ? __uint_as_float(v[j]) + __uint_as_float(x[j]) : __uint_as_float(v[j]));
                        }
                    }
                }
            } else if (alive) {
                ptx::tc_fence_after();
                const int blocks = (P.BN / 32 + 1) / 2; // whole 32-column blocks per set
                with_store_mode(store_mode(), J.res != nullptr, [&](auto mode_c, auto res_c) {
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
                            r[h + j] = SPLIT ? __uint_as_float(v[j]) + __uint_as_float(x[j]) : __uint_as_float(v[j]);
                    }
                    store_block<decltype(mode_c)::value, decltype(res_c)::value>(J, r, stage, f_tile0 + c);
                }
                });
            }
        }
    } else if (warp >= kDrainWarp) {
        // ---------------- drain warps: running totals of flushed accumulators; persistent mode: the epilogue ----------------
        ptx::reg_alloc<Regs<PP>::drain>();
        const int quarter = warp & 3, p = quarter * 32 + lane, FL = SPLIT ? P.fl : 0;
        const int n_groups = FL > 0 ? (KS + FL - 1) / FL : 1;
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
            auto drain = [&](auto mode_c, auto res_c) {
            [[maybe_unused]] constexpr int MODE = decltype(mode_c)::value; // (a single tile stores nothing here)
            [[maybe_unused]] constexpr bool RES = decltype(res_c)::value;
            for (int tl = 0; tl < ntl && alive; ++tl) {
                const int reg = two_regions ? (tl & 1) : 0, use = two_regions ? (tl >> 1) : tl;
                StoreJob J;
                if (PP) { // where the tile goes: worked out while its MMAs run
                    set_tile((int)blockIdx.x + tl * (int)gridDim.x);
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
                    alive = ptx::mbar_wait_warp(reg ? acc_full1 : acc_full, (uint32_t)(use & 1), abort_flag);
                    ptx::tc_fence_after();
                };
                auto release = [&]() { // the MMA thread may start the region's next tile
                    ptx::tc_fence_before();
                    __syncwarp();
                    if (lane == 0)
                        ptx::mbar_arrive(acc_empty + reg);
                };
                if constexpr (PP == kNarrow) {
                    take_acc_full();
                    if (!alive)
                        break;
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
                                racc[h + j] = SPLIT ? __uint_as_float(v[j]) + __uint_as_float(x[j]) : __uint_as_float(v[j]);
                        }
                        if (c + 32 >= P.BN)
                            release();
                        store_block<MODE, RES>(J, racc, stage, ntile * P.BN + c);
                    }
                } else {
                    // Groups in order, round-to-nearest adds; the MMA thread restarts the main accumulator once a group has been taken.
                    for (int g = 0; g + 1 < n_groups && alive; ++g, gpar ^= 1u) {
                        alive = ptx::mbar_wait_warp(acc_ready, gpar, abort_flag);
                        if (!alive)
                            break;
                        ptx::tc_fence_after();
                        drain_add<false>(racc, tmain, 0u, P.BN, g == 0);
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
                        drain_add<false>(racc, tmain, 0u, P.BN, n_groups == 1);
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
                        drain_add<SPLIT>(racc, tmain, tcross, P.BN, n_groups == 1);
                        release();
#pragma unroll 1
                        for (int c = 0; c < P.BN; c += 32) {
                            store_block<MODE, RES>(J, racc, stage, ntile * P.BN + c);
#pragma unroll
                            for (int j = 0; j < 96; ++j) // the next block's sums move down
                                racc[j] = racc[j + 32];
                        }
                    }
                }
            }
            };
            if constexpr (PP == kSingle)
                drain(std::integral_constant<int, kStoreAny>(), std::integral_constant<bool, false>()); // (stores nothing)
            else
                with_store_mode(store_mode(), P.res != nullptr, drain);
            if (!PP && FL > 0) // (also after a wait gave up: the transform sets wait here)
                ptx::named_bar_sync(1, 384);
        }
    }

    // ---------------- split-K: reduction across the cluster ----------------
    // Every thread of every CTA of the cluster reaches the barrier (all waits above are bounded).
    if (P.ksplit > 1) {
        if (warp >= kSetWarp && warp < kSetWarp + 4) {
            // The bias / residual values the reduction below adds start their way to L1 while the cluster meets.  Set 0's
            // threads do it, for the row each of them wrote into sYoff itself (both halves of the CTA's column slice).
            const int et = threadIdx.x - kSetWarp * 32, cols = P.BN / P.ksplit;
            const long long y_off = sYoff[et];
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
            const long long y_off = sYoff[et & (kTileM - 1)];
            if (y_off >= 0 && *abort_flag == 0) {
                const long long f_glob0 = P.z_is_batch ? 0 : (long long)zb * P.Fg;
                float *yp = P.y + y_off + f_glob0 * P.ys_f;
                const float *bp = P.has_bias ? P.bias + f_glob0 : nullptr;
                const float *rp = P.res != nullptr ? P.res + y_off + f_glob0 * P.ys_f : nullptr;
                const int rank = (int)ptx::cluster_ctarank();
                // 16-byte stores need filters contiguous in y, 16-byte aligned rows, and column runs of at least 2
                const bool red_vec = (P.ys_f == 1) && ((P.ys_p & 3) == 0) && ((P.ys_n & 3) == 0) && ((P.Fg & 3) == 0) &&
                                     ((reinterpret_cast<uintptr_t>(P.y) & 15) == 0) && (P.BN / P.ksplit >= 4) &&
                                     (P.res == nullptr || (reinterpret_cast<uintptr_t>(P.res) & 15) == 0);
#define PETB200_RED(ACT_) \
    cluster_reduce_store<ACT_>(sSplit, P.ksplit, rank, P.BN, et, ntile * P.BN, P.Fg, bp, rp, yp, P.ys_f, red_vec)
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
    if (*abort_flag) {
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

// -------------------------------------------------------------------------------------------------------------
// weight packing: W[F][cpg][T] (conv) or B[b][k][n] / B[b][n][k] (matmul) -> hi/lo [rows][Ktot], K ordered as the
// kernel consumes it: k = chunk*Kc_pad + tap*BC + ci, zero where there is no such element.
// -------------------------------------------------------------------------------------------------------------
// hi/lo parts of one packed value: TF32 (hi = top 19 bits, or rounded for a single pass) as fp32 words, or bf16 halves
template <bool BF> __device__ __forceinline__ void store_split(void *hi, void *lo, long long i, float v, int rna) {
    if (BF) {
        const uint32_t h = ptx::pack_bf16x2(v, 0.f) & 0xffffu;
        reinterpret_cast<uint16_t *>(hi)[i] = (uint16_t)h;
        reinterpret_cast<uint16_t *>(lo)[i] = (uint16_t)(ptx::pack_bf16x2(v - __uint_as_float(h << 16), 0.f) & 0xffffu);
    } else {
        const float h = rna ? __uint_as_float(ptx::cvt_rna_tf32(v)) : __uint_as_float(__float_as_uint(v) & 0xffffe000u);
        reinterpret_cast<float *>(hi)[i] = h;
        reinterpret_cast<float *>(lo)[i] = v - h;
    }
}

template <bool BF>
__global__ void __launch_bounds__(256) k_pack_conv_w(const float *__restrict__ w, void *__restrict__ hi,
                                                     void *__restrict__ lo, int F, int cpg, int T, int BC, int Kc_pad,
                                                     int nchunks, int rna) {
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
        store_split<BF>(hi, lo, i, v, rna);
    }
}

// What a matmul needs before it can run, in one launch (bound by HBM: every operand read once, its copy written once).
// Blocks [0, b_tiles): B[b][k][n] or [b][n][k] -> hi/lo [rows][Kpad], a tile of 32 rows x 32 packed positions per block; a [k][n]
// tile is turned through shared memory, so that both sides move whole 128-byte lines (one thread per packed position read B
// with a stride of n words: 35 us of the 76 us of a 4 x 500 x 1001 x 770 product).  The other blocks: rows of A copied to a
// pitch that TMA can address (the padding is zero).
struct PrepareArgs {
    const float *b;
    void *hi, *lo;
    int bs, n, k, Kpad, rna, BC;
    FastDiv by_kc_pad, by_tiles_k, by_tiles_n;
    long long sb_batch, sb_row;
    int b_tiles, tiles_k, tiles_n;
    const float *a;
    float *a_copy;
    long long a_rows;
    int a_w, a_pitch;
};
template <bool BF, bool TRANSB>
__global__ void __launch_bounds__(256) k_prepare_mm(const PrepareArgs g) {
    pdl_prologue();
    __shared__ float tile[32][33];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if ((int)blockIdx.x >= g.b_tiles) { // rows of A, a warp each
        const long long stride = (long long)(gridDim.x - g.b_tiles) * 8;
        for (long long r = (long long)(blockIdx.x - g.b_tiles) * 8 + warp; r < g.a_rows; r += stride) {
            const float *src = g.a + r * g.a_w;
            float *dst = g.a_copy + r * g.a_pitch;
#pragma unroll 8
            for (int c = lane; c < g.a_pitch; c += 32)
                dst[c] = c < g.a_w ? __ldg(src + c) : 0.f;
        }
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
                store_split<BF>(g.hi, g.lo, ((long long)bb * g.n + nn) * g.Kpad + k0 + lane, v, g.rna);
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
                store_split<BF>(g.hi, g.lo, ((long long)bb * g.n + nn) * g.Kpad + k0 + lane, tile[lane][warp + i], g.rna);
        }
    }
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

typedef void (*KernelFn)(CUtensorMap, CUtensorMap, CUtensorMap, IgemmParams);

struct TcCore {
    int beside = 1; // launches of this size that share the GPU (a split of K then only adds work)
    petb200_ctx *ctx = nullptr;
    IgemmParams P{};
    int single_pass = 0;
    int bf16 = 0; // error-compensated bf16 (64 K elements per stage) instead of TF32
    dim3 grid;
    size_t smem = 0;
    // geometry needed to (re)encode the activation map
    int xd[5]{}; // W,H,D,C,N of the activation tensor as the kernel sees it
    long long a_row = 0, a_batch = 0; // row-major matmul A: element strides of a row and of a batch entry
    long long Ktot = 0;
    int rows_b = 0;
    DevBuf whi, wlo, koff;
    long long y_elems = 0;
    CUtensorMap map_x{}, map_bhi{}, map_blo{};
    const void *map_x_ptr = nullptr;
    bool weights_ready = false;
    int starve = 0;

    KernelFn kernel() const {
        if (P.a_kmajor && P.band_w > 0) // banded products: G2BMM in persistent mode with its own epilogue, GBMML with its own operand fetch
            return P.band_g2 ? k_igemm<true, kMathTf32x3, kNarrow, 1>
                             : (!P.pp ? k_igemm<true, kMathTf32x3, kSingle, 2>
                                      : (P.BN <= 64 && P.fl == 0 ? k_igemm<true, kMathTf32x3, kNarrow, 2> : k_igemm<true, kMathTf32x3, kWide, 2>));
        if (single_pass)
            return pick<kMathTf32x1>();
        return bf16 ? pick<kMathBf16x3>() : pick<kMathTf32x3>();
    }
    template <int PASSES> KernelFn pick() const {
        const bool narrow = P.BN <= 64 && P.fl == 0;
        if (P.a_kmajor)
            return !P.pp ? k_igemm<true, PASSES> : (narrow ? k_igemm<true, PASSES, kNarrow> : k_igemm<true, PASSES, kWide>);
        return !P.pp ? k_igemm<false, PASSES> : (narrow ? k_igemm<false, PASSES, kNarrow> : k_igemm<false, PASSES, kWide>);
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
    int encode_b() {
        EncodeTiledFn enc = encode_fn();
        if (!enc)
            return fail(ctx, PETB200_ERR_CUDA, "cuTensorMapEncodeTiled entry point unavailable");
        cuuint64_t dims[2] = {(cuuint64_t)Ktot, (cuuint64_t)rows_b};
        cuuint64_t str[1] = {(cuuint64_t)Ktot * (bf16 ? 2 : 4)};
        cuuint32_t box[2] = {(cuuint32_t)P.ke, (cuuint32_t)P.BN}; // one 128-byte row of K per filter
        cuuint32_t es[2] = {1, 1};
        for (int i = 0; i < 2; ++i) {
            CUresult r = enc(i ? &map_blo : &map_bhi, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2,
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
        IgemmParams p = P;
        set_divisors(p);
        p.link = link;
        p.bias = bias;
        p.res = res;
        p.y = y;
        p.koff = (const int *)koff.p;
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
static int cluster_slots(int sm_count, int ks) {
    static int cached[17] = {0};
    if (ks <= 1)
        return sm_count;
    if (cached[ks] == 0) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(1, (unsigned)ks * 64, 1);
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = 200 * 1024; // enough that two CTAs never share an SM, as in every real plan
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 1, attr[0].val.clusterDim.y = (unsigned)ks, attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr, cfg.numAttrs = 1;
        int n = 0;
        (void)cudaFuncSetAttribute(k_igemm<false, kMathTf32x3>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (ks > 8) // clusters of 16 are beyond the portable size: allowed per function
            (void)cudaFuncSetAttribute(k_igemm<false, kMathTf32x3>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (cudaOccupancyMaxActiveClusters(&n, k_igemm<false, kMathTf32x3>, &cfg) != cudaSuccess || n <= 0) {
            (void)cudaGetLastError();
            // what B200 was measured to hold; a cluster of 16 is only used where the driver itself says it fits
            n = ks > 8 ? -1 : std::max(1, (sm_count * (ks <= 2 ? 96 : 86) / 100) / ks);
        }
        cached[ks] = n;
    }
    return cached[ks];
}

// Rough cycle model of one launch, used to pick the tile width and the K split.  A K stage is charged its MMAs (N/2 cycles each,
// 12 per stage for 3xTF32, 4 for one pass) or 520 cycles, a CTA 3000 cycles before its first MMA and 1700 + 44*BN of epilogue
// (split-K: the exchange through the cluster instead), every wave of CTAs the sum.
// These constants rank the choices; they don't predict times.  With persistent tiles, where start-up and epilogue hide, a 3xTF32
// stage was measured to take about 1000 cycles at 128 filters (charged 768), 690 at 64 and 570 at 32 (charged 520).  Against the
// fastest of all (width, split) pairs, forced one by one, on 44 shapes (every convolution of ResNet-18 at batch 1, 8 and 64 and
// of ResNet3D-18, the 512-channel dilated one, the projections of an encoder of 768 at 128 and 384 rows), the choice is
// within 2 % on 38.  The other six lose 6 to 34 % because 128-filter tiles, five times with K split in two, are preferred to unsplit
// 64-filter ones: 64 -> 128 channels at stride 2 (batch 8: 15.7 us against 11.8; 1x1 at batch 64: 26.6 against 19.9; 3-D:
// 29.4 against 26.5), 128 -> 128 at batch 8 (19.5 against 18.4), 384 rows of 768 -> 2304 and 3072 (15.4 against 12.5).
static double est_cycles(int sm_count, long long base_ctas, int nchunks, int spc, int BN, int passes, int ks) {
    const double stage = std::max<double>((passes == 3 ? 12.0 : 4.0) * (BN / 2), 520.0);
    const long long stages = (long long)((nchunks + ks - 1) / ks) * spc;
    // split-K: (ks-1)/ks of the 512*BN-byte tile crosses to other SMs at ~10 bytes per cycle, then barrier + local sums
    const double per_cta = 3000.0 + (double)stages * stage + 1700.0 + (ks > 1 ? 1500.0 + 50.0 * BN * (ks - 1) / ks : 44.0 * BN);
    const long long slots = cluster_slots(sm_count, ks);
    if (slots <= 0)
        return 1e30; // this cluster size cannot be launched here
    const long long waves = (base_ctas + slots - 1) / slots;
    return (double)waves * per_cta;
}
// Split K over 1, 2, 4, 8 or 16 CTAs (a cluster; 16 is beyond the portable cluster size and allowed per function): the
// split must divide the tile width and leave every CTA a chunk.
static int choose_ksplit(int sm_count, long long base_ctas, const IgemmParams &P, int passes, int want, double *cycles) {
    auto ok = [&](int ks) { return ks == 1 || (ks <= P.nchunks && P.BN % ks == 0); };
    int best = 1;
    double best_c = est_cycles(sm_count, base_ctas, P.nchunks, P.spc, P.BN, passes, 1);
    static const int ks_cap = std::min(16, std::max(1, env_int_early("PETB200_TC_KSPLIT_MAX", 16)));
    if (want > 0) {
        for (best = 16; best > 1 && !(best <= want && ok(best) && cluster_slots(sm_count, best) > 0); best /= 2) {
        }
        best_c = est_cycles(sm_count, base_ctas, P.nchunks, P.spc, P.BN, passes, best);
    } else {
        for (int ks = 2; ks <= ks_cap; ks *= 2) {
            if (!ok(ks))
                continue;
            const double c = est_cycles(sm_count, base_ctas, P.nchunks, P.spc, P.BN, passes, ks);
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
    // (bf16: twice the K per stage and an accuracy class that the split, not the truncation, dominates: half as often)
    const int period = env_int("PETB200_TC_FLUSH", core.bf16 ? 16 : 8);
    const int ks_max = ((P.nchunks + P.ksplit - 1) / P.ksplit) * P.spc;
    P.fl = (!core.single_pass && period > 0 && ks_max > 3 * period) ? period : 0;
    if (env_int("PETB200_TC_VERBOSE", 0))
        fprintf(stderr, "[petb200] igemm plan: BN %d BC %d chunks %d stages/chunk %d ksplit %d flush %d NB %d NR %d kmajor %d flat %d math %s\n",
                P.BN, P.BC, P.nchunks, P.spc, P.ksplit, P.fl, P.NB, P.NR, P.a_kmajor, P.flat,
                core.single_pass ? "1xtf32" : (core.bf16 ? "bf16x3" : "3xtf32"));
}

// Persistent mode (see IgemmParams::pp) where some SM would otherwise run several CTAs in sequence: the start-up of a CTA (about
// 3000 cycles to its first MMA) and its epilogue (2000 to 4000) hide behind the MMAs of its neighbour tiles.  Not with a K
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

// The dynamic shared-memory attribute is per function, not per launch: raise it once to the device limit so that plans
// with different needs can coexist.
static int raise_smem_limit(petb200_ctx *ctx) {
    static bool attr_set = false;
    if (attr_set)
        return PETB200_OK;
    const int lim = (int)std::min<size_t>(ctx->smem_optin, 227 * 1024);
    const KernelFn kernels[] = {
        k_igemm<false, kMathTf32x3>, k_igemm<false, kMathTf32x3, kNarrow>, k_igemm<false, kMathTf32x3, kWide>,
        k_igemm<true, kMathTf32x3>, k_igemm<true, kMathTf32x3, kNarrow>, k_igemm<true, kMathTf32x3, kWide>,
        k_igemm<false, kMathTf32x1>, k_igemm<false, kMathTf32x1, kNarrow>, k_igemm<false, kMathTf32x1, kWide>,
        k_igemm<true, kMathTf32x1>, k_igemm<true, kMathTf32x1, kNarrow>, k_igemm<true, kMathTf32x1, kWide>,
        k_igemm<false, kMathBf16x3>, k_igemm<false, kMathBf16x3, kNarrow>, k_igemm<false, kMathBf16x3, kWide>,
        k_igemm<true, kMathBf16x3>, k_igemm<true, kMathBf16x3, kNarrow>, k_igemm<true, kMathBf16x3, kWide>,
        k_igemm<true, kMathTf32x3, kNarrow, 1>, k_igemm<true, kMathTf32x3, kSingle, 2>, k_igemm<true, kMathTf32x3, kNarrow, 2>,
        k_igemm<true, kMathTf32x3, kWide, 2>};
    cudaError_t e = cudaSuccess;
    for (auto k : kernels)
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
    if (e != cudaSuccess)
        return fail(ctx, PETB200_ERR_CUDA, "cudaFuncSetAttribute(%d bytes) failed: %s", lim, cudaGetErrorString(e));
    attr_set = true;
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
    P.ke = core.bf16 ? 64 : kStageK;
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
        const long long base_ctas = (long long)mtiles * ((Fg + bn - 1) / bn) * gz * core.beside;
        const int passes = core.single_pass ? 1 : 3;
        double cyc;
        const int ks = choose_ksplit(ctx->sm_count, base_ctas, P, passes, want_ks, &cyc);
        if (ks > 1) { // the landing area takes shared memory from the rings (or even from the chunk size): fit again
            P.ksplit = ks;
            if (!fit(bn))
                continue;
            if (P.nchunks < ks) {
                P.ksplit = 1;
                if (!fit(bn))
                    continue;
                cyc = est_cycles(ctx->sm_count, base_ctas, P.nchunks, P.spc, bn, passes, 1);
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
    if (core.koff.alloc(koff.size() * 4) != cudaSuccess)
        return fail(ctx, PETB200_ERR_NOMEM, "koff allocation failed");
    PETB200_CUDA(ctx, cudaMemcpy(core.koff.p, koff.data(), koff.size() * 4, cudaMemcpyHostToDevice));
    return raise_smem_limit(ctx);
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
    t->full.single_pass = passes == kMathTf32x1;
    t->full.bf16 = passes == kMathBf16x3;
    const long long plane = (long long)g.OD * g.OH * g.OW;
    t->ys[0] = (long long)g.F * plane;
    t->ys[1] = channels_last_out ? 1 : plane;
    t->ys[2] = channels_last_out ? g.F : 1;
    // Rows that are not multiples of 16 bytes cannot be a TMA stride: small planes are fetched whole ("flat"), anything
    // else is re-pitched by the caller first (tc_conv_row_pitch tells it to what).
    int rc = PETB200_ERR_UNSUPPORTED;
    if (g.W % 4 != 0) {
        rc = tc_configure(ctx, t->full, g, 0, g.OH, 0, g.OW, 0, g.N, t->ys[0], t->ys[1], t->ys[2], has_bias, act, 0, 0, 0, 1);
        if (rc == PETB200_ERR_UNSUPPORTED) {
            g.Wst = (g.W + 3) / 4 * 4;
            memset(&t->full.P, 0, sizeof t->full.P);
        }
    }
    if (rc == PETB200_ERR_UNSUPPORTED)
        rc = tc_configure(ctx, t->full, g, 0, g.OH, 0, g.OW, 0, g.N, t->ys[0], t->ys[1], t->ys[2], has_bias, act);
    if (rc) {
        delete t;
        return rc;
    }
    TcCore &c = t->full;
    c.rows_b = g.F;
    size_t wbytes = (size_t)g.F * c.Ktot * (c.bf16 ? 2 : 4);
    if (c.whi.alloc(wbytes) != cudaSuccess || c.wlo.alloc(wbytes) != cudaSuccess) {
        delete t;
        return fail(ctx, PETB200_ERR_NOMEM, "packed weight allocation (%zu bytes) failed", 2 * wbytes);
    }
    rc = c.encode_b();
    if (rc) {
        delete t;
        return rc;
    }
    *dev_bytes = 2 * wbytes + c.koff.bytes;
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
    t->full.single_pass = passes == kMathTf32x1;
    t->full.bf16 = passes == kMathBf16x3;
    t->full.beside = beside;
    t->ys[0] = ys_n, t->ys[1] = ys_f, t->ys[2] = ys_p;
    int rc = PETB200_ERR_UNSUPPORTED;
    if (w % 4 != 0)
        rc = tc_configure(ctx, t->full, g, 0, ohn, 0, own, 0, n, ys_n, ys_f, ys_p, has_bias, act, 0, 0, 0, 1);
    else
        rc = tc_configure(ctx, t->full, g, 0, ohn, 0, own, 0, n, ys_n, ys_f, ys_p, has_bias, act);
    if (rc) {
        delete t;
        return rc;
    }
    TcCore &core = t->full;
    core.rows_b = f;
    const size_t wbytes = (size_t)f * core.Ktot * (core.bf16 ? 2 : 4);
    if (core.whi.alloc(wbytes) != cudaSuccess || core.wlo.alloc(wbytes) != cudaSuccess) {
        delete t;
        return fail(ctx, PETB200_ERR_NOMEM, "packed weight allocation (%zu bytes) failed", 2 * wbytes);
    }
    rc = core.encode_b();
    if (rc) {
        delete t;
        return rc;
    }
    *dev_bytes = 2 * wbytes + core.koff.bytes;
    *out = t;
    return PETB200_OK;
}

void tc_conv_destroy(void *h) { delete (TcConv *)h; }

int tc_conv_set_weights(void *h, const float *w, cudaStream_t s) {
    auto *t = (TcConv *)h;
    TcCore &c = t->full;
    const int cpg = t->g.C / t->g.groups, T = t->g.T3[0] * t->g.T3[1] * t->g.T3[2];
    long long total = (long long)t->g.F * c.Ktot;
    int blocks = (int)std::min<long long>((total + 255) / 256, (long long)c.ctx->sm_count * 16);
    if (c.bf16)
        k_pack_conv_w<true><<<blocks, 256, 0, s>>>(w, c.whi.p, c.wlo.p, t->g.F, cpg, T, c.P.BC, c.P.spc * c.P.ke, c.P.nchunks, 0);
    else
        k_pack_conv_w<false><<<blocks, 256, 0, s>>>(w, c.whi.p, c.wlo.p, t->g.F, cpg, T, c.P.BC, c.P.spc * c.P.ke, c.P.nchunks,
                                                    c.single_pass);
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
        wc->single_pass = t->full.single_pass;
        wc->bf16 = t->full.bf16;
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
    return cudaMemcpyToSymbol(ptx::g_mbar_wait_limit_ns, &ns, sizeof ns) == cudaSuccess ? PETB200_OK : PETB200_ERR_CUDA;
}
int tc_conv_row_pitch(void *h) { return ((TcConv *)h)->g.Wst; }
const char *tc_conv_variant(void *h) {
    const TcCore &c = ((TcConv *)h)->full;
    return c.single_pass ? "tc_1xtf32_ts" : (c.bf16 ? "tc_bf16x3_ts" : "tc_3xtf32_ts");
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
    P.ke = core.bf16 ? 64 : kStageK;
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
            const int ks = choose_ksplit(ctx->sm_count, (long long)P.tpi * ((n + bn - 1) / bn) * bs, P, core.single_pass ? 1 : 3,
                                         env_int("PETB200_TC_KSPLIT", 0), &cyc);
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
    if (core.koff.alloc(koff.size() * 4) != cudaSuccess)
        return fail(ctx, PETB200_ERR_NOMEM, "koff allocation failed");
    PETB200_CUDA(ctx, cudaMemcpy(core.koff.p, koff.data(), koff.size() * 4, cudaMemcpyHostToDevice));
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
    t->core.single_pass = passes == kMathTf32x1;
    t->core.bf16 = passes == kMathBf16x3;
    const long long dense[6] = {(long long)m * k, transA ? m : k, (long long)k * n, transB ? k : n, (long long)m * n, n};
    for (int i = 0; i < 6; ++i)
        t->st[i] = strides ? strides[i] : dense[i];
    int rc;
    if (!transA && k % 4 == 0 && t->st[0] % 4 == 0 && t->st[1] % 4 == 0) {
        rc = tc_configure_kmajor(ctx, t->core, bs, m, n, k, has_bias, act, t->st);
    } else if (!transA && !strides) { // rows of A off the 16-byte grid: the same on a copy with a pitch of whole 16-byte pieces
        t->a_rows = (long long)bs * m, t->a_w = k, t->a_pitch = (k + 3) / 4 * 4;
        const long long st[6] = {(long long)m * t->a_pitch, t->a_pitch, t->st[2], t->st[3], t->st[4], t->st[5]};
        rc = tc_configure_kmajor(ctx, t->core, bs, m, n, t->a_pitch, has_bias, act, st);
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
        rc = tc_configure(ctx, t->core, g, 0, 1, 0, m, 1, bs, (long long)m * n, 1, n, has_bias, act);
    }
    if (rc) {
        delete t;
        return rc;
    }
    TcCore &c = t->core;
    c.rows_b = bs * n;
    // rows of different batch entries are adjacent: Fg = n rows per z
    size_t wbytes = (size_t)bs * n * c.Ktot * (c.bf16 ? 2 : 4);
    if (c.whi.alloc(wbytes) != cudaSuccess || c.wlo.alloc(wbytes) != cudaSuccess) {
        delete t;
        return fail(ctx, PETB200_ERR_NOMEM, "packed B allocation failed");
    }
    rc = c.encode_b();
    if (rc) {
        delete t;
        return rc;
    }
    *dev_bytes = 2 * wbytes + c.koff.bytes;
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
    std::vector<int> koff(P.ke, -1);
    if (core.koff.alloc(koff.size() * 4) != cudaSuccess) {
        delete t;
        return fail(ctx, PETB200_ERR_NOMEM, "koff allocation failed");
    }
    cudaMemcpy(core.koff.p, koff.data(), koff.size() * 4, cudaMemcpyHostToDevice);
    core.grid = dim3((unsigned)std::min(P.tiles, ctx->sm_count), 1u, 1u);
    core.y_elems = (long long)bs * n * (2 * w + 1);
    core.rows_b = bs * n;
    const size_t wbytes = (size_t)bs * n * core.Ktot * 4;
    int rc = raise_smem_limit(ctx);
    if (rc == PETB200_OK && (core.whi.alloc(wbytes) != cudaSuccess || core.wlo.alloc(wbytes) != cudaSuccess))
        rc = fail(ctx, PETB200_ERR_NOMEM, "packed key allocation failed");
    if (rc == PETB200_OK)
        rc = core.encode_b();
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
    std::vector<int> koff(P.spc * P.ke, -1);
    if (core.koff.alloc(koff.size() * 4) != cudaSuccess) {
        delete t;
        return fail(ctx, PETB200_ERR_NOMEM, "koff allocation failed");
    }
    cudaMemcpy(core.koff.p, koff.data(), koff.size() * 4, cudaMemcpyHostToDevice);
    core.y_elems = (long long)bs * n * m;
    core.rows_b = bs * m;
    const size_t wbytes = (size_t)bs * m * core.Ktot * 4;
    int rc = raise_smem_limit(ctx);
    if (rc == PETB200_OK && (core.whi.alloc(wbytes) != cudaSuccess || core.wlo.alloc(wbytes) != cudaSuccess))
        rc = fail(ctx, PETB200_ERR_NOMEM, "packed value allocation failed");
    if (rc == PETB200_OK)
        rc = core.encode_b();
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
void tc_matmul_destroy(void *h) { delete (TcMatmul *)h; }
// Packs B (null: it has been) and copies A to an addressable pitch (null: not needed), in one launch.
int tc_matmul_prepare(void *h, const float *b, const float *a, float *a_copy, cudaStream_t s) {
    auto *t = (TcMatmul *)h;
    TcCore &c = t->core;
    PrepareArgs g{};
    g.b = b, g.hi = c.whi.p, g.lo = c.wlo.p, g.bs = t->bs, g.n = t->n, g.k = t->k, g.Kpad = (int)c.Ktot, g.rna = c.single_pass;
    g.BC = c.P.BC, g.sb_batch = t->st[2], g.sb_row = t->st[3];
    g.tiles_k = g.Kpad / 32, g.tiles_n = (t->n + 31) / 32; // (Kpad is a multiple of 32)
    g.by_kc_pad.set(c.P.spc * c.P.ke), g.by_tiles_k.set(g.tiles_k), g.by_tiles_n.set(g.tiles_n);
    const long long tiles = b ? (long long)g.tiles_k * g.tiles_n * t->bs : 0;
    if (tiles > (1 << 30))
        return fail(c.ctx, PETB200_ERR_UNSUPPORTED, "matmul operand too large to pack in one launch");
    g.b_tiles = (int)tiles;
    g.a = a, g.a_copy = a_copy, g.a_rows = a ? t->a_rows : 0, g.a_w = t->a_w, g.a_pitch = t->a_pitch;
    const long long a_blocks = std::min<long long>((g.a_rows + 7) / 8, (long long)c.ctx->sm_count * 8);
    if (tiles + a_blocks == 0)
        return PETB200_OK;
    const dim3 grid((unsigned)(tiles + a_blocks));
    if (c.bf16)
        launch_pdl(t->transB ? k_prepare_mm<true, true> : k_prepare_mm<true, false>, grid, 256, 0, s, g);
    else
        launch_pdl(t->transB ? k_prepare_mm<false, true> : k_prepare_mm<false, false>, grid, 256, 0, s, g);
    if (b)
        c.weights_ready = true;
    return launched(c.ctx, "k_prepare_mm");
}
int tc_matmul_pack_b(void *h, const float *b, cudaStream_t s) { return tc_matmul_prepare(h, b, nullptr, nullptr, s); }
int tc_matmul_run(void *h, const float *a_t, const float *bias, const float *res, float *cmat, cudaStream_t s) {
    auto *t = (TcMatmul *)h;
    return t->core.launch(a_t, bias, res, cmat, s);
}

} // namespace petb200
