// Tiled mixed-precision collocate / integrate.
//
// Persistent CTAs take work units from an atomic queue.  A unit is one tile of
// one grid level (TX x TY x TZ points, x fastest; TX = 32, TY x TZ = 128 rows with
// TZ = 4 or 8 per level, chosen by the tile autotuner) with its items, the periodic
// images of pairs whose sphere reaches it, or a part of that list for the busiest
// tiles and at the queue's end (those units flush with atomics).  The pair records,
// coefficients and images are copied one item ahead with cp.async.  Per item:
//   1-D tables t^k exp(-zetp t^2) over the tile's three ranges   (float-float)
//   stage 1  Cxy[z][b][a] = sum_g c[g][b][a] Z[g][z]              (float-float)
//   stage 2  Cx[(z,y)][a] = sum_b Cxy[z][b][a] Y[b][y]            (float-float)
//   stage 3  rho[(z,y)][x] = sum_a Cx[(z,y)][a] X[a][x]           (exact fp16 slices)
// (the three contractions of collocate_core, collocate.cc:543-623, with the
// cube culling of grid_collocate_core, grid_base_ref_c.cc:413-471).
//
// Stage 3 operands are split into NSL fixed-point fp16 slices of SLB bits: each
// row of Cx is scaled by a power of two so its largest entry is < 2^SLB, each
// column of X likewise, and the slices are integers (the first in [-2^SLB,
// 2^SLB], the others in [-2^(SLB-1), 2^(SLB-1)]).  They carry the float-float
// operand to ~2^-35 of its row's scale (its low part enters through one float32
// remainder).  Every slice product is an integer of at most 2^20, so the
// anti-diagonal sums D_s = sum over i+j=s of A_i B_j are exact in FP32 for the
// leading two (16 and 32 products, at most 2^24); the next two (48 and 64 products)
// can pass 2^24 only in the worst case, where their
// rounding stays below 2^-40 of the scales.  (Integrate contracts 32 x: D2 is
// kept as two K halves of 16 products; its D3 sums 64 and can round in the worst
// case, by less than 2^-35 of the scales.)  The diagonals are recombined in
// float-float.  The tile sum
// over pairs is float-float (high parts in registers, low parts in shared
// memory), added to the FP64 grid once per tile.
//
// Integrate is the transpose: S[(z,y)][a] = sum_x V[(z,y)][x] X[a][x] by the same
// slices (V sliced once per unit into the A operand, each item masking its rows there
// and restoring them from a per-CTA global slot that stays in L2), then the adjoint
// stages, and the per-pair moments are added to FP64 scratch with atomics.
//
// General (non-orthorhombic) cells use the same kernels instantiated with
// kGeneral (t_d along the lattice steps, the quadratic row rule, the Gaussian's
// cross factor per point) when their level has a tile shape; by default they
// run on the float-float general kernel (gpw_fp64.cu).
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <string>
#include <vector>

#include "gpw_coef.cuh"
#include "gpw_ff.cuh"
#include "gpw_internal.h"
#include "gpw_tc.cuh"

namespace gpw {

constexpr int TX = 32;
constexpr int MROWS = 128;       // TY * TZ rows per tile, one per thread
constexpr int kMaxTY = 32, kMaxTZ = 8;  // tiles of 32 x 16 x 8 or 32 x 32 x 4
constexpr int kMaxTZColl = 8;  // collocate keeps its stage-1 output for at most 8 z (tiles with TZ <= 8)
static_assert(kMaxTZ <= kMaxTZColl, "tile shapes that collocate holds");
constexpr int NTHR = MROWS;
constexpr int NSL = 4;          // slices per operand
constexpr int SLB = 10;         // bits per slice
constexpr int KP = 16;          // padded contraction length (alpha)
constexpr int NCOEF_MAX = ((kMaxLp + 1) * (kMaxLp + 2) * (kMaxLp + 3)) / 6;

// Periodic images of one axis of a cube over one tile.  Every image is an item of its
// own, so the limit only bounds their number: a cube far larger than its cell has some
// k^3 images over each tile (500 pairs with cubes of 10 cells a side on a 16^3 grid:
// 678,000 items, 42 MB).  The binning leaves such a pair out, and tiled calls report it.
constexpr int kMaxImages = 4;

struct TileDesc {
    int level;
    int t[3];  // tile indices
    int lz;    // log2 TZ (TY = MROWS >> lz)
    int flags; // kUnitSplit
};

// the tile's pairs are divided among several work units: flush with atomics
constexpr int kUnitSplit = 1;

// tile extents of a tile descriptor
struct TileShape {
    int TY, TZ, ly, lz;
    __host__ __device__ explicit TileShape(int lz_) : TY(MROWS >> lz_), TZ(1 << lz_), ly(7 - lz_), lz(lz_) {}
};

// ---------------------------------------------------------------------------
// pair data a tile needs, staged in shared memory
struct TPair {
    double r2;          // radius^2 (FP64, rule decisions)
    double hz, hy, hx;  // spacings (orthorhombic rule); general cell: 1 / |v_2|, 1 / |v_1|, 1 / |v_0|
    float r2f, hzf, hyf, hxf;
    float hyinvf, hxinvf;  // 1/hy, 1/hx rounded to float
    ff zetp;
    ff off[3];          // roffset
    ff h[3];
    int lb[3], hi[3], cc[3];
    int kgmin, lp, L;
    float gpf[3];       // general: gp - cc as FP32 (once per pair: FP64 conversions per row are slow)
    int general;        // general cell: box-relative cube (lb = 0), lattice-step lengths in h
    int64_t coef_off, table_off;
    double gp[3];       // general: the product centre in lattice coordinates (dh_inv^T rp)
    double radius;      // general: the cube radius (the row rule squares it itself)
};
// General-cell level constants of the tiled path: FP32 lattice steps for the row
// rule, and the cosines between the steps (cross terms of the Gaussian).
struct GenLevel {
    GeneralRow32 row;
    GeneralRowFF rowff;
    ff c01, c02, c12;   // cos(v0, v1), cos(v0, v2), cos(v1, v2)
};
// The sphere of a general-cell pair in the tiled path.  On tiled levels sum t_d^2 <=
// 2.5 r^2 (mixed_build), so the cross factor at a point is at most exp(1.5 zetp r^2): it
// must not leave float's range, nor dwarf the row's other points, whose slices share one
// scale.  Points beyond zetp r^2 = 46, below 1e-20 of the Gaussian's peak, are left out (radii
// from eps = 1e-10 give 23).
constexpr double kMaxExponent = 46.0;
__device__ __forceinline__ double tiled_radius(const PairGeom &g) {
    return fmin(g.radius, sqrt(kMaxExponent / g.zetp));
}
// A pair's blob: the record padded to kHdr16 16-byte chunks, then its
// coefficients as float-float (written by every collocate call), padded to 16 bytes.
constexpr int kHdr16 = (int)((sizeof(TPair) + 15) / 16);
constexpr int kCoef16Max = (NCOEF_MAX * (int)sizeof(float2) + 15) / 16;

// one periodic image of a pair over the tile
struct ImgState {
    ff tc;              // collocate: x of the re-expansion column minus xp
    int o[3];           // cube offset of the tile origin
    int gx0, gx1;       // tile-local x range inside the cube box
    int ic;             // collocate: tile-local re-expansion column
    int sb;             // collocate: x-variable scale 2^sb of the slices (balancing)
};

// Per (tile, pair image) item, computed once per task set: the image's state.  A
// cube that reaches a tile through several periodic images (small cells) has one
// item per image, each kept only if its own sphere reaches the tile.  (Before, one
// item that the kernels looped over, every combination of the axes' images a full
// pass: 1000 pairs, l <= 2, in a 10-bohr cell, 64^3, took 0.94 ms to collocate; with
// items per image and shorter units 0.36 ms.)
struct alignas(16) ItemImg {
    ImgState im;
    int pad_;
};
static_assert(sizeof(ItemImg) == 48, "ItemImg is three 16-byte chunks");

struct MixedState {
    int ntiles = 0;
    int64_t nitems = 0;
    TileDesc *d_tiles = nullptr;
    uint4 *d_blob = nullptr;       // pair blobs of the orthorhombic tasks (sorted order)
    int64_t *d_blob_off = nullptr; // per task: blob offset in 16-byte chunks
    int64_t *d_start = nullptr;    // per work unit: first item, end
    uint64_t *d_items = nullptr;   // per (tile, pair image): blob offset << 16 | chunks
    ItemImg *d_iimg = nullptr;     // per item: its image
    int *d_queue = nullptr;      // [0]: collocate, [1]: integrate (orthorhombic tiles), [2], [3]: general tiles
    GenLevel *d_glv = nullptr;   // per level (general levels only meaningful)
    int northo = 0;              // ortho tasks come first in sorted order
    int64_t nbin = 0;            // tasks [0, nbin) are binned (the ortho ones, then general ones if tiled)
    bool gen_tiled = false;      // general-cell pairs run on the tiled kernels
    int ntiles_ortho = 0;        // tiles [0, ntiles_ortho) are orthorhombic, the rest general
    int sms = 0;
    int per_sm = 0, per_sm_i = 0, per_sm_ig = 0;  // resident CTAs: collocate, integrate (ortho, general)
    uint4 *d_vslot = nullptr, *own_vslot = nullptr;  // integrate: per-CTA V slots, in the scratch memory or their own
    // binning state kept for re-binning on the device (gpw_taskset_update_geometry)
    std::vector<TileDesc> h_tiles;  // every tile of the binned levels, in tile-index order
    struct BinLevel *d_bl = nullptr;  // per level: first tile index, tiles per axis, tile shape
    int *d_blob_len = nullptr;      // per binned pair: chunks of its blob
    int *d_count = nullptr;         // per tile: items; then whether pairs were left out (kMaxImages)
    bool over = false;              // the last binning's
    unsigned long long *d_cursor = nullptr;  // per tile: next item slot (fill pass)
    unsigned char *d_units = nullptr;        // d_cursor, d_start and d_tiles, one after the other
    int64_t cap_items = 0, cap_units = 0;    // capacities of d_items / d_iimg, and of d_units in bytes
};


// ---------------------------------------------------------------------------
// Sphere rule (FP32 with an error bound, fast_floor_checked in gpw_common.cuh).
// the exact FP64 rule, out of line: taken only where the FP32 estimate is unsure;
// the row's imax, or -1 for a row outside the cube
__device__ __noinline__ int rule_row_exact(const TPair &p, int kf, int jf) {
    const double remk = rule_remk(p.r2, kf, p.hz);
    return jf < -rule_jmax(remk, p.hy) ? -1 : rule_imax(remk, jf, p.hy, p.hx);
}

// imax of the folded row (kf, jf), negative outside the cube.  The row lies in the
// cube when (jf hy)^2 <= r^2 - (kf hz)^2: the sign of the remainder decides it, away
// from zero by more than its error bound.
__device__ __forceinline__ int row_imax(const TPair &p, int kf, int jf) {
    const float dz = (float)(-kf) * p.hzf, dy = (float)(-jf) * p.hyf;
    const float rem = __fmaf_rn(-dy, dy, __fmaf_rn(-dz, dz, p.r2f));
    if (rem < p.r2f * -4.8e-7f) return -1;
    bool unsure;
    const int i = fast_floor_checked(rem, p.r2f, p.hxinvf, unsure);
    return unsure ? rule_row_exact(p, kf, jf) : i;
}

// Row (z, y) of the tile: cube-local x range [x0, x1] (empty if x0 > x1).
__device__ __forceinline__ void row_range(const TPair &p, const ImgState &q, const int *table, int gz, int gy,
                                          int ext_ok, int &x0, int &x1) {
    x0 = 1;
    x1 = 0;
    if (!ext_ok || gz < p.lb[2] || gz > p.hi[2] || gy < p.lb[1] || gy > p.hi[1]) return;
    const int kf = fold(gz), jf = fold(gy);
    if (kf < p.kgmin) return;
    int imin;
    if (p.table_off < 0) {
        imin = -row_imax(p, kf, jf);
        if (imin > 0) return;
    } else {
        const int *T = table + p.table_off;
        const int kidx = kf - T[0];
        const int jmin = T[1 + 2 * kidx];
        if (jf < jmin) return;
        imin = T[1 + 2 * (1 - T[0]) + T[2 + 2 * kidx] + (jf - jmin)];
    }
    // cube offsets [imin, 1 - imin] -> tile-local
    x0 = max(imin - q.o[0], q.gx0);
    x1 = min(1 - imin - q.o[0], q.gx1);
}

// General cell: the row (jj, kk) of the index box holds the points i with
// |i v0 + w|^2 <= r^2 (the reference's quadratic, grid_base_ref_c.cc:781-807; FP32 with
// an error bound, then float-float, then FP64).
__device__ __forceinline__ bool general_row_fast(const LevelDev &lv, const GenLevel &G, const TPair &p, int jj,
                                                 int kk, int &ismin, int &ismax) {
    bool unsure;
    const bool some = general_row_fast32(G.row, p.gpf[0], p.gpf[1], p.gpf[2], (float)(jj - p.cc[1]) - p.gpf[1],
                                         (float)(kk - p.cc[2]) - p.gpf[2], p.r2f, p.cc[0], ismin, ismax, unsure);
    if (!unsure) return some;
    return general_row_unsure(&G.rowff, lv.dh, p.gp, p.cc[0], jj, kk, p.radius, ismin, ismax);
}

// Row (z, y) of the tile for a general-cell pair: tile-local x range [x0, x1].
__device__ __forceinline__ void general_row_range(const LevelDev &lv, const GenLevel &G, const TPair &p,
                                                  const ImgState &q, int gz, int gy, int ext_ok, int &x0,
                                                  int &x1) {
    x0 = 1;
    x1 = 0;
    if (!ext_ok || gz < 0 || gz > p.hi[2] || gy < 0 || gy > p.hi[1]) return;
    int ismin, ismax;
    if (!general_row_fast(lv, G, p, p.cc[1] + gy, p.cc[2] + gz, ismin, ismax)) return;
    x0 = max(ismin - p.cc[0] - q.o[0], q.gx0);
    x1 = min(ismax - p.cc[0] - q.o[0], q.gx1);
}

// UMMA canonical K-major layout, no swizzle: core matrices of 8 rows x 16 bytes
// (8 halves of K).  Element (row r, k) of an operand with R rows, K = 16:
//   byte offset = (r / 8) * SBO + (k / 8) * LBO + (r % 8) * 16 + (k % 8) * 2,
// LBO = 128 (next 8 K-elements), SBO = 256 (next 8 rows).

constexpr int kZeroExp = -1000;
// 2^k as a float, -126 <= k <= 127
__device__ __forceinline__ float pow2i(int k) { return __int_as_float((127 + k) << 23); }
// e with m = f 2^e, f in [0.5, 1); values below 2^-100 count as zero
__device__ __forceinline__ int exp_of(float m) {
    return m >= 7.888609052210118e-31f ? ((__float_as_int(m) >> 23) & 0xff) - 126 : kZeroExp;
}
// the NSL fixed-point slices of two values v * scale, scale = 2^(SLB - e)
__device__ __forceinline__ void slice_scaled2(ff2 v, float2 scale, float2 *sl) {
    const float2 hi = f2_mul(v.hi, scale), lo = f2_mul(v.lo, scale);
    sl[0] = f2_rint(hi);
    float2 r = f2_add(f2_sub(hi, sl[0]), lo);
#pragma unroll
    for (int i = 1; i < NSL; i++) {
        r = f2_mul(r, f2(1024.0f));
        sl[i] = f2_rint(r);
        r = f2_sub(r, sl[i]);
    }
}
// two slices (integers of at most 2^SLB) as packed halves
__device__ __forceinline__ uint32_t pack_halves(float2 s) {
    const __half2 h2 = __floats2half2_rn(s.x, s.y);
    return *reinterpret_cast<const uint32_t *>(&h2);
}

struct MixedArgs {
    const uint4 *blob;        // per pair: record (kHdr16 chunks) then float-float coefficients
    const LevelDev *levels;
    const TileDesc *tiles;
    const int64_t *start;
    const uint64_t *items;    // per (tile, pair image): blob offset in 16-byte chunks << 16 | chunks to copy
    const ItemImg *iimg;      // per item: its image
    const int *table;
    const GenLevel *glv;  // general levels: FP32 steps, cosines
    double *mom;  // integrate: per-pair moments
    uint4 *vslot;  // integrate: one slot of kVSlot16 chunks per CTA (the tile's V)
    GridPtrs grids;
    int *queue;
    int *status;
    int ntiles;
};

// one pair as staged in shared memory: the record, then its coefficients
// (collocate only), in the blob's own layout so that it is copied chunk by chunk
struct alignas(16) PairBuf {
    union {
        TPair p;
        uint4 hdr_[kHdr16];
    };
    float2 coef[2 * kCoef16Max];
};
// the record alone (integrate)
struct alignas(16) PairHdr {
    union {
        TPair p;
        uint4 hdr_[kHdr16];
    };
};

// shared state of both tiled kernels
struct TileCommon {
    ItemImg ii[2];  // the image of the current item and of the one being fetched
    int tile;
    float2 exptab[32];  // c_exp2_32: the lanes' indices differ, a constant-bank read would be replayed per value
    uint64_t mbar;
    uint32_t tmem;
    int abort;
};

// Cxy rows b (L - b values of a) padded to an even length: start of row b
__host__ __device__ constexpr int cxy_pad_row(int L, int b) {
    int q = 0;
    for (int i = 0; i < b; i++) q += (L - i + 1) & ~1;
    return q;
}
constexpr int kNPair = (kNPow + 1) / 2;                     // pairs of a
constexpr int kCxyRow = cxy_pad_row(kNPow, kNPow) / 2;      // 16-byte entries of one z

// Collocate's re-expansion and stage 1 have one output per thread and turn, each the end
// of a chain of up to lp + 1 steps: the outputs in order of falling chain length, so that
// the lanes of a warp have chains of about one length (re-expansion at lp = 8: in packed
// order a warp's longest chain was 2.4 times the mean of all, in this order 1.4 times).
struct Order {
    uint32_t rec[d_decode_at(kNPow)];       // per lp: g | b << 4 | a << 8 | packed index << 16
    unsigned char st1[kNPow][2 * kCxyRow];  // [L - 1]: b | a << 4, the padding of rows as well
};
constexpr Order make_order() {
    Order o{};
    for (int lp = 0; lp < kNPow; lp++) {
        int at = d_decode_at(lp);
        for (int d = 0; d <= lp; d++) {  // chain length lp + 1 - d
            int t = 0;
            for (int g = 0; g <= lp; g++)
                for (int b = 0; b <= lp - g; b++)
                    for (int a = 0; a <= lp - g - b; a++, t++)
                        if (g + b + a == d) o.rec[at++] = (uint32_t)(g | b << 4 | a << 8 | t << 16);
        }
        at = 0;
        for (int d = 0; d <= lp + 1; d++) {  // d = lp + 1: the padding, no terms
            for (int b = 0; b <= lp; b++)
                for (int a = 0; a < ((lp - b + 2) & ~1); a++)
                    if (a + b == d) o.st1[lp][at++] = (unsigned char)(b | a << 4);
        }
    }
    return o;
}
static __device__ const Order d_order = make_order();

struct alignas(128) SmemColl {
    __half A[NSL][MROWS * KP];  // Cx slices, M=128 x K=16
    __half B[NSL][TX * KP];     // X slices, N=32 x K=16
    ff rc[NCOEF_MAX];           // coefficients re-expanded around the tile's column ic
    float4 Cxy[kMaxTZColl][kCxyRow];  // stage 1 output, pairs of a: {hi, hi, lo, lo}
    PairBuf pb[2];              // the current pair and the one being fetched
    ff Y[kNPow][kMaxTY + 1];  // rows padded: lanes reading different rows hit different banks
    // the z table for packed products of two z: high parts, and both parts negated
    alignas(16) float Zh[kNPow][kMaxTZ], Znh[kNPow][kMaxTZ], Znl[kNPow][kMaxTZ];
    alignas(16) float acc_lo[MROWS][TX + 4];  // low parts of the tile sums (row m belongs to thread m; padded rows)
    float bin[kNPow][kNPow];    // binomials C(a', a) of the re-expansion
    unsigned char st1[kNPow][2 * kCxyRow];  // d_order.st1
    alignas(16) float cs[2][TX];  // 2^fx per column (0 for an empty column), of this item and the next
    TileCommon c;
};

static_assert(4 * (sizeof(SmemColl) + 1024) <= 228 * 1024, "4 collocate CTAs per SM");

// Integrate keeps the tile's V in a 32 KB per-CTA global slot that stays in L2.
// Orthorhombic: V's slices stand in the A operand; each pair zeroes what lies outside its
// rows' ranges, and restores it afterwards from the slot, a copy of the slices in the A
// operand's layout (both K halves).  General cells rescale the rows per image: A is built
// anew from V as float-float in the slot, [x pair][row], read one 16-byte chunk group
// ahead.  (With V in shared memory three CTAs fitted an SM, and S and T had to share the
// operands' memory: 7.47 ms for 8000 pairs on 128^3, 7.13 with four.)
constexpr int kVSlot16 = 2 * NSL * MROWS * KP / 8;

// Integrate's tables and sums for packed products of four y or z (16-byte loads):
// Y[b][y] in three planes; S[alpha][(z,y)] and T[(b,a)][z] in two, rows of S padded so
// that the lanes' different alpha fall into different banks.
constexpr int kYRow = kMaxTY + 4;
constexpr int kSRow = MROWS + 4;
struct IntSums {
    alignas(16) float Sh[kNPow][kSRow], Sl[kNPow][kSRow];
};
// Integrate's B operand (N = 16 alpha x K = 16 x per half, per slice): core
// matrices 160 bytes apart along K and 288 along N, the second K half 64 bytes
// further on.  Warp 0 stores one alpha row at a time, lane (h, k) the 2-byte
// element (alpha, k) of half h: the four groups of 8 lanes (h, k / 8) then fill
// four disjoint sets of 4 banks (the dense layout, 128 and 2048 bytes apart, put
// all four into the same banks).
constexpr int kBLbo = 160, kBSbo = 288, kBPlane = 576;       // bytes
constexpr int kBHalf = NSL * kBPlane + 64;                   // bytes from half 0 to half 1
__host__ __device__ constexpr int b_off(int row, int k) {    // bytes within a plane
    return (row >> 3) * kBSbo + (k >> 3) * kBLbo + (row & 7) * 16 + (k & 7) * 2;
}
static_assert(b_off(15, 15) + 2 <= kBPlane && kBPlane % 16 == 0 && kBHalf % 16 == 0, "B planes");
static_assert(kBPlane == 2 * kBSbo, "the planes follow one another along N");

struct alignas(128) SmemInt {
    alignas(16) float Yh[kNPow][kYRow], Ynl[kNPow][kYRow];
    alignas(8) float gsc[KP];                // 2^(g - SLB), g the alpha row's exponent (0: an empty row)
    PairHdr pb[2];                           // the current pair's record and the one being fetched
    TileCommon c;
    alignas(16) float Ynh[kNPow][kYRow];
    alignas(16) float Zh[2][kNPow][kMaxTZ], Znl[2][kNPow][kMaxTZ];  // of this item and the next
    uint32_t mask[MROWS];          // orthorhombic: each row's points inside the item's range
    uint8_t todo[MROWS];           // the chunks of its A row to be masked to them
    __half A[2][NSL][MROWS * KP];  // slices of V (times the cross factor), K halves x in [0,16) and [16,32)
    IntSums st;                    // S, then T in the columns of S that a warp is done with
    alignas(16) unsigned char B[2 * kBHalf];  // X' slices: plane (h, q) at h kBHalf + q kBPlane
};
// planes of the y table: none (collocate: float-float entries), high and negated low, and -Y.hi
template <class Smem>
constexpr int kYPlanes = 3;
template <>
constexpr int kYPlanes<SmemColl> = 0;
// dynamic shared memory of integrate: more than 46 KB, so that no fifth CTA (for which
// TMEM has no columns left) is placed on an SM
static_assert(4 * (sizeof(SmemInt) + 1024) <= 228 * 1024, "4 integrate CTAs per SM");
static_assert(5 * (sizeof(SmemInt) + 1024) > 228 * 1024, "at most 4 integrate CTAs per SM");

// ---- asynchronous record copies (cp.async, 16-byte chunks, L2 only)
__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tc::smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Starts copying item it into buf / ii: the pair's record, its coefficients when
// with_coef, and the item's images.  Each thread waits for its own copies
// (cp_async_wait_all) before the barrier after which the buffers are read.
__device__ __forceinline__ void fetch_pair(uint4 *dst, ItemImg &ii, const MixedArgs &A, int64_t it, uint64_t item,
                                           bool with_coef) {
    const uint4 *src = A.blob + (item >> 16);
    const int n = with_coef ? min((int)(item & 0xFFFFu), kHdr16 + kCoef16Max) : kHdr16;
    const uint4 *isrc = reinterpret_cast<const uint4 *>(A.iimg + it);
    // dst: the record's chunks, the coefficients following without a gap
    uint4 *idst = reinterpret_cast<uint4 *>(&ii);
    for (int t = threadIdx.x; t < n + 3; t += blockDim.x) {
        if (t < n) cp_async16(dst + t, src + t);
        else cp_async16(idst + (t - n), isrc + (t - n));
    }
    cp_async_commit();
}

__device__ __forceinline__ void set_image_x(const TPair &p, ImgState &q, int ox, int ext_x) {
    q.o[0] = ox;
    q.gx0 = max(0, p.lb[0] - ox);
    q.gx1 = min(ext_x - 1, p.hi[0] - ox);
    // Re-expansion column: start from the column nearest to the product centre and
    // move toward the tile centre by at most one Gaussian width 1/sqrt(zetp) --
    // the largest values stay near u = 0, and broad Gaussians get the smallest
    // |u| over the whole tile.
    const float hx = p.h[0].hi;
    int i0 = (int)rintf(__fdividef(p.off[0].hi, hx)) - ox;  // any column is valid: approximate
    i0 = min(max(i0, q.gx0), max(q.gx0, q.gx1));
    const float rg = rsqrtf(p.zetp.hi) / hx;
    const float dc = fminf(fmaxf((float)(TX / 2 - i0), -rg), rg);
    q.ic = i0 + (int)rintf(dc);
    q.tc = ff_add(ff_mul_f(p.h[0], (float)(ox + q.ic)), ff{-p.off[0].hi, -p.off[0].lo});
    // Balance the powers: u -> u / 2^sb with 2^sb ~ the extent that matters on this
    // tile, min(max |u|, 2 / sqrt(zetp)); the row coefficients take 2^(k sb), so the
    // product is unchanged and both operands' slices keep their bits where the
    // values are.
    const float umax = (float)max(q.ic - q.gx0, q.gx1 - q.ic) * hx;
    const float ext = fminf(umax, 2.0f * rsqrtf(p.zetp.hi));
    const int e = ((__float_as_int(ext) >> 23) & 0xff) - 126;  // ext = f 2^e, f in [0.5, 1)
    q.sb = ext >= 1.1754944e-38f ? min(max(e, -10), 10) : 0;
}
// tab[k][i] = u^k exp(-zetp t^2), t = g h - off, g = o + i, and u = t or, for x
// with recentre, u = (i - ic) h / 2^sb (the balanced offset from the
// re-expansion column); zero outside the cube box, outside the valid tile extent
// and for k >= L.
//
// One entry per lane: warp 0 entry x of the x column (kept in registers), warp 1
// entry ent of the y table (ent < TY) or of the z table.  In collocate both warps
// run one loop over entries, so that the kernel holds a single copy of the
// float-float exponential, its largest inlined function: collocate is limited by
// instruction fetch, and this alone took it from 995 to 926 ms per launch on the
// 1M-pair workload.
struct TileExt {
    int x, y, z;  // the tile's points inside the grid, per axis
};
struct TabEntry {
    ff t, e;    // t = g h - off and exp(-zetp t^2) (zero outside)
    int d, i;   // axis and tile-local index
    bool in;    // inside the cube box and the tile's valid extent
};
__device__ __forceinline__ TabEntry tab_entry(const TPair &p, const ImgState &q, const TileExt &ext,
                                              const TileShape &sh, const float2 *exptab, int warp, int ent) {
    TabEntry r;
    const bool isy = ent < sh.TY;
    r.d = warp == 0 ? 0 : (isy ? 1 : 2);
    r.i = warp == 0 || isy ? ent : ent - sh.TY;
    const int g = q.o[r.d] + r.i;
    r.in = r.i < (warp == 0 ? ext.x : (isy ? ext.y : ext.z)) && g >= p.lb[r.d] && g <= p.hi[r.d];
    r.t = ff_add(ff_mul_f(p.h[r.d], (float)g), ff{-p.off[r.d].hi, -p.off[r.d].lo});
    r.e = r.in ? ff_exp(ff_mul(ff_mul(r.t, r.t), ff{-p.zetp.hi, -p.zetp.lo}), exptab) : ff{0.0f, 0.0f};
    return r;
}
// warp 1: one y or z entry's powers: Y as float-float entries (collocate) or, as Z, in
// three planes (high parts, both parts negated) for packed products
template <class Smem>
__device__ __forceinline__ void yz_fill(Smem &sm, const TPair &p, const TabEntry &te, int zbuf) {
    constexpr int kY = kYPlanes<Smem>;
    const bool isy = te.d == 1;
    const int L = te.in ? p.L : 0;
    ff e = te.e;
    if constexpr (kY == 0) {
        float *hi = isy ? &sm.Y[0][te.i].hi : &sm.Zh[0][te.i], *lo = isy ? hi + 1 : &sm.Znl[0][te.i];
        const int stride = isy ? 2 * (kMaxTY + 1) : kMaxTZ;
        float *nhi = &sm.Znh[0][te.i];
        const float sg = isy ? 1.0f : -1.0f;
#pragma unroll 1
        for (int k = 0; k < p.L; k++) {  // (to kNPow: 61.0 -> 62.2 ms, 100k pairs, 256^3)
            hi[k * stride] = k < L ? e.hi : 0.0f;
            lo[k * stride] = k < L ? sg * e.lo : 0.0f;
            if (!isy) nhi[k * stride] = k < L ? -e.hi : 0.0f;
            e = ff_mul(e, te.t);
        }
    } else {
        float *hi = isy ? &sm.Yh[0][te.i] : &sm.Zh[zbuf][0][te.i];
        float *nlo = isy ? &sm.Ynl[0][te.i] : &sm.Znl[zbuf][0][te.i], *nhi = &sm.Ynh[0][te.i];
        const int stride = isy ? kYRow : kMaxTZ;
#pragma unroll 1
        for (int k = 0; k < p.L; k++) {
            hi[k * stride] = k < L ? e.hi : 0.0f;
            if (isy) nhi[k * stride] = k < L ? -e.hi : 0.0f;
            nlo[k * stride] = k < L ? -e.lo : 0.0f;
            e = ff_mul(e, te.t);
        }
    }
}
// Binomials C(a', a) of the re-expansion c'[g][b][a] = sum_{a' >= a} C(a', a)
// tc^(a' - a) c[g][b][a'] around column ic of the tile: powers of the small
// offsets u = x - x_ic keep the stage-3 operands well conditioned for the
// fixed-point slices.
__constant__ float c_binom[kNPow][kNPow] = {
    {1},
    {1, 1},
    {1, 2, 1},
    {1, 3, 3, 1},
    {1, 4, 6, 4, 1},
    {1, 5, 10, 10, 5, 1},
    {1, 6, 15, 20, 15, 6, 1},
    {1, 7, 21, 35, 35, 21, 7, 1},
    {1, 8, 28, 56, 70, 56, 28, 8, 1},
    {1, 9, 36, 84, 126, 126, 84, 36, 9, 1},
    {1, 10, 45, 120, 210, 252, 210, 120, 45, 10, 1}};

// c_zs[lp][g]: packed index of (g, 0, 0)
#define GPW_ZS(lp) {ZS_(lp, 0), ZS_(lp, 1), ZS_(lp, 2), ZS_(lp, 3), ZS_(lp, 4), ZS_(lp, 5), ZS_(lp, 6), ZS_(lp, 7), ZS_(lp, 8), ZS_(lp, 9), ZS_(lp, 10), ZS_(lp, 11)}
#define ZS_(lp, g) ((g) > (lp) + 1 ? 0 : (((lp) + 1) * ((lp) + 2) * ((lp) + 3) - ((lp) + 1 - (g)) * ((lp) + 2 - (g)) * ((lp) + 3 - (g))) / 6)
__constant__ int c_zs[kNPow][kNPow + 1] = {GPW_ZS(0), GPW_ZS(1), GPW_ZS(2), GPW_ZS(3), GPW_ZS(4), GPW_ZS(5),
                                           GPW_ZS(6), GPW_ZS(7), GPW_ZS(8), GPW_ZS(9), GPW_ZS(10)};
#undef ZS_
#undef GPW_ZS

// One item (g, b, a) per thread of [t0, t0 + nt): Horner in tc over a' = amax .. a
// with the binomials from shared memory (bin[a'][a] = C(a', a)).  The row coefficients'
// balancing factor 2^(a sb) is applied here, once per coefficient.
__device__ void recentre_x(const PairBuf &pb, ff tc, int sb, ff *out, const float (*bin)[kNPow], int t0, int nt) {
    const int lp = pb.p.lp;
    const int nc = ncoef(lp);
    for (int i = (int)threadIdx.x - t0; i < nc; i += nt) {
        const uint32_t de = __ldg(&d_order.rec[d_decode_at(lp) + i]);
        const int g = de & 15, b = (de >> 4) & 15, a = (de >> 8) & 15, t = de >> 16, amax = lp - g - b;
        const int base = t - a;  // packed index of (g, b, 0)
        ff s = {0.0f, 0.0f};
#pragma unroll 1
        for (int ap = amax; ap >= a; ap--) {
            const float2 c = pb.coef[base + ap];
            s = ff_fma(s, tc, ff_mul_f(ff{c.x, c.y}, bin[ap][a]));
        }
        const float bal = pow2i(a * sb);  // balancing of the x powers (exact)
        out[t] = ff{__fmul_rn(s.hi, bal), __fmul_rn(s.lo, bal)};
    }
}

// masks of the 8 packed halves of one 16-byte chunk from bits 0..7 of b (bit k:
// half k, all ones or zero).  One multiply per 4 bits moves bit k to the top of
// byte k (the copies lie 7 bits apart, so no carries), and prmt, whose selector
// nibbles with the top bit set replicate the sign of the selected byte, spreads
// each byte's top bit over the two bytes of its half.
__device__ __forceinline__ uint4 chunk_mask(uint32_t b) {
    const uint32_t lo = ((b & 0xFu) * 0x10204080u) & 0x80808080u;
    const uint32_t hi = (((b >> 4) & 0xFu) * 0x10204080u) & 0x80808080u;
    uint4 m;
    asm("prmt.b32 %0, %1, 0, 0x9988;" : "=r"(m.x) : "r"(lo));
    asm("prmt.b32 %0, %1, 0, 0xBBAA;" : "=r"(m.y) : "r"(lo));
    asm("prmt.b32 %0, %1, 0, 0x9988;" : "=r"(m.z) : "r"(hi));
    asm("prmt.b32 %0, %1, 0, 0xBBAA;" : "=r"(m.w) : "r"(hi));
    return m;
}

// The NSL slices of one K = 16 operand row (v[i]: the values 2 i and 2 i + 1, zero
// beyond kNPow), scaled by sc, as 16-byte chunks of 8 K values in the UMMA layout
// (planes of plane_halves halves); K groups at or beyond kw are left as they are, and
// those at or beyond nval (only zeros there) are written as zeros directly.
__device__ __forceinline__ void slice_row16(const ff2 *vin, float sc, int kw, int nval, __half *plane0,
                                            int plane_halves, int row) {
    // one compact loop body for both K groups: the second group's values are moved down
    ff2 v[4];
#pragma unroll
    for (int i = 0; i < 4; i++) v[i] = vin[i];
#pragma unroll 1
    for (int kg = 0; kg < KP / 8; kg++) {
        if (8 * kg >= kw) break;
        const int o16 = (row >> 3) * 16 + kg * 8 + (row & 7);  // offset of (row, 8 kg) / 16
        if (8 * kg >= nval) {  // only zeros left: rewrite the stale slots without slicing
#pragma unroll
            for (int q = 0; q < NSL; q++) reinterpret_cast<uint4 *>(plane0 + q * plane_halves)[o16] = make_uint4(0, 0, 0, 0);
            continue;
        }
        uint32_t w[NSL][4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            float2 sl[NSL];
            slice_scaled2(v[i], f2(sc), sl);
#pragma unroll
            for (int q = 0; q < NSL; q++) w[q][i] = pack_halves(sl[q]);
        }
#pragma unroll
        for (int q = 0; q < NSL; q++)
            reinterpret_cast<uint4 *>(plane0 + q * plane_halves)[o16] = make_uint4(w[q][0], w[q][1], w[q][2], w[q][3]);
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = 4 + i < kNPair ? vin[4 + i < kNPair ? 4 + i : 0] : ff2{f2(0.0f), f2(0.0f)};
    }
}

// General cell: the cross factor along row (z, y) of the current image, E(x) =
// exp(alpha + beta t0(x)) with beta = -2 zetp (c01 t1 + c02 t2), alpha = -2 zetp
// c12 t1 t2: returns E of the pair of x (even, odd) that holds the row's first cube point
// x0, and what next_cross needs.  Outside the cube's points E may leave float's range, so
// no value comes from outside: where x0 is the odd one the even one is not used.
__device__ __forceinline__ void cross_factor_row(const GenLevel &G, const TPair &P, const ImgState &Q,
                                                 const float2 *exptab, int z, int y, int x0, ff2 &e, ff2n &qn) {
    const ff t1 = ff_add(ff_mul_f(P.h[1], (float)(Q.o[1] + y)), ff{-P.off[1].hi, -P.off[1].lo});
    const ff t2 = ff_add(ff_mul_f(P.h[2], (float)(Q.o[2] + z)), ff{-P.off[2].hi, -P.off[2].lo});
    const ff t0 = ff_add(ff_mul_f(P.h[0], (float)(Q.o[0] + x0)), ff{-P.off[0].hi, -P.off[0].lo});
    const ff m2z = {-2.0f * P.zetp.hi, -2.0f * P.zetp.lo};
    const ff beta = ff_mul(m2z, ff_add(ff_mul(G.c01, t1), ff_mul(G.c02, t2)));
    const ff alpha = ff_mul(m2z, ff_mul(G.c12, ff_mul(t1, t2)));
    const ff2 eq = ff2_exp(ff2_pair(ff_add(alpha, ff_mul(beta, t0)), ff_mul(beta, P.h[0])), exptab);
    const ff e0 = {eq.hi.x, eq.lo.x}, q = {eq.hi.y, eq.lo.y};
    e = ff2_pair(e0, x0 & 1 ? e0 : ff_mul(e0, q));
    qn = ff2n_of(ff2_pair(q, ff_mul(q, q)));
}
// the next pair's, from the odd one: E q, E q^2
__device__ __forceinline__ ff2 next_cross(ff2 e, ff2n q) { return ff2_mul(ff2_dup(ff{e.hi.y, e.lo.y}), q); }

// General cell, integrate: the A operand row r = the slices of V(x) E(x) over the
// row's cube points [x0, x1] (zero elsewhere), with the row's own exponent (returned).
// V (float-float, two x per 16 bytes) comes from the CTA's slot, 8 x ahead of their use.
template <class Smem>
__device__ __forceinline__ int general_a_row(Smem &sm, const uint4 *vslot, const GenLevel &G, const TPair &P,
                                             const ImgState &Q, const TileShape &sh, int r, int x0, int x1) {
    if (x0 > x1) return kZeroExp;  // the row's products are not read
    const float4 *const vrow = reinterpret_cast<const float4 *>(vslot) + r;
    ff2 e0;
    ff2n q;
    const int xs = x0 & ~1;  // two x per instruction
    float4 nx[4];
#pragma unroll
    for (int i = 0; i < 4; i++) nx[i] = vrow[(4 * (xs >> 3) + i) * MROWS];
    cross_factor_row(G, P, Q, sm.c.exptab, r >> sh.ly, r & (sh.TY - 1), x0, e0, q);
    // pass 1: the row maximum of |V E|, of which only the exponent counts: leading parts alone
    // (a value may exceed the scale by 2^-19 of it, which the first slice absorbs)
    float mx = 0.0f;
    {
        float2 e = e0.hi;
#pragma unroll 1
        for (int c = xs >> 3; 8 * c <= x1; c++) {
            float4 v4[4];
            const int cn = 8 * (c + 1) <= x1 ? c + 1 : 0;
#pragma unroll
            for (int i = 0; i < 4; i++) v4[i] = nx[i];
#pragma unroll
            for (int i = 0; i < 4; i++) nx[i] = vrow[(4 * cn + i) * MROWS];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int x = 8 * c + 2 * i;
                if (x >= xs && x <= x1) {
                    const float2 v = f2_mul(make_float2(v4[i].x, v4[i].z), e);
                    if (x >= x0) mx = fmaxf(mx, fabsf(v.x));
                    if (x < x1) mx = fmaxf(mx, fabsf(v.y));
                    e = f2_mul(f2(e.y), q.hi);
                }
            }
        }
    }
    const int vmx = exp_of(mx);
    const float sc = vmx == kZeroExp ? 0.0f : pow2i(SLB - vmx);
    // pass 2: slices, 16-byte chunks of 8 x
    ff2 e = e0;
#pragma unroll 1
    for (int c = 0; c < TX / 8; c++) {
        uint32_t w[NSL][4];
        float4 v4[4];
#pragma unroll
        for (int i = 0; i < 4; i++) v4[i] = nx[i];
        if (c < TX / 8 - 1) {
#pragma unroll
            for (int i = 0; i < 4; i++) nx[i] = vrow[(4 * c + 4 + i) * MROWS];
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int x = 8 * c + 2 * i;
            ff2 v = {f2(0.0f), f2(0.0f)};
            if (x >= xs && x <= x1) {
                v = ff2_mul(ff2{make_float2(v4[i].x, v4[i].z), make_float2(v4[i].y, v4[i].w)}, ff2n_of(e));
                if (x < x0) v.hi.x = v.lo.x = 0.0f;
                if (x == x1) v.hi.y = v.lo.y = 0.0f;
                e = next_cross(e, q);
            }
            float2 sl[NSL];
            slice_scaled2(v, f2(sc), sl);
#pragma unroll
            for (int qq = 0; qq < NSL; qq++) w[qq][i] = pack_halves(sl[qq]);
        }
        const int o16 = (r >> 3) * 16 + (c & 1) * 8 + (r & 7);
#pragma unroll
        for (int qq = 0; qq < NSL; qq++)
            reinterpret_cast<uint4 *>(sm.A[c >> 1][qq])[o16] = make_uint4(w[qq][0], w[qq][1], w[qq][2], w[qq][3]);
    }
    return vmx;
}

// Orthorhombic integrate: the A row r to the points of M (bit x) in its chunks of 8 x
// that hold more than those (bits of todo).
template <class Smem>
__device__ __forceinline__ void mask_a_row(Smem &sm, int r, uint32_t M, uint32_t todo) {
#pragma unroll
    for (int v = 0; v < TX / 8; v++) {
        if (!((todo >> v) & 1u)) continue;
        const uint4 mk = chunk_mask((M >> (8 * v)) & 0xFFu);
        uint4 *a = reinterpret_cast<uint4 *>(sm.A[v >> 1][0]) + (r >> 3) * 16 + (v & 1) * 8 + (r & 7);
        uint4 t[NSL];
#pragma unroll
        for (int q = 0; q < NSL; q++) t[q] = a[q * (MROWS * KP / 8)];
#pragma unroll
        for (int q = 0; q < NSL; q++)
            a[q * (MROWS * KP / 8)] = make_uint4(t[q].x & mk.x, t[q].y & mk.y, t[q].z & mk.z, t[q].w & mk.w);
    }
}
// Copies from the CTA's slot the chunks of row r in which the next item (mask M) needs
// points that the row no longer holds (asynchronously: waited for at the item's end);
// returns what the row then holds.
template <class Smem>
__device__ __forceinline__ uint32_t restore_a_row(Smem &sm, const uint4 *vslot, int r, uint32_t M, uint32_t have) {
    // chunk v of slice q lies a constant away from the row's first chunk, in both copies
    const uint32_t dst = tc::smem_addr(sm.A) + 16 * ((r >> 3) * 16 + (r & 7));
    const uint4 *src = vslot + (r >> 3) * 16 + (r & 7);
    const uint32_t lack = M & ~have;
    if (lack != 0u) {
#pragma unroll
        for (int v = 0; v < TX / 8; v++) {
            if (((lack >> (8 * v)) & 0xFFu) == 0u) continue;
            have |= 0xFFu << (8 * v);
#pragma unroll
            for (int q = 0; q < NSL; q++) {
                const int o = ((v >> 1) * NSL + q) * (MROWS * KP / 8) + (v & 1) * 8;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * o), "l"(src + o) : "memory");
            }
        }
    }
    cp_async_commit();
    return have;
}
// the chunks (bits 0..3) of a row holding the points `have` that an item with the points M
// masks; none in a row without points: its products are not read
__device__ __forceinline__ uint8_t chunks_to_mask(uint32_t M, uint32_t have) {
    const uint32_t d = __vcmpne4(M, have) & 0x08040201u;  // a byte per chunk
    return M == 0u ? 0 : (uint8_t)((d | d >> 8 | d >> 16 | d >> 24) & 15u);
}
// bits x0..x1 of a row's cube range in the item (P, Q)
__device__ __forceinline__ uint32_t row_mask(const TPair &P, const ImgState &Q, const int *table, int z, int y, bool ok) {
    int x0, x1;
    row_range(P, Q, table, Q.o[2] + z, Q.o[1] + y, ok, x0, x1);
    return x0 > x1 ? 0u : (uint32_t)(((2ull << x1) - 1ull) & ~((1ull << x0) - 1ull));
}

// TMEM set-up shared by both kernels: warp 0 allocates, thread 0 inits the mbarrier
__device__ __forceinline__ void tc_setup(TileCommon &c, uint32_t ncols) {
    if (threadIdx.x == 0) {
        tc::mbar_init(&c.mbar, 1);
        tc::fence_mbar_init();
        c.abort = 0;
    }
    if (threadIdx.x < 32) {
        c.exptab[threadIdx.x] = c_exp2_32[threadIdx.x];
        tc::tmem_alloc(&c.tmem, ncols);
        tc::tmem_relinquish();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
}

__device__ __forceinline__ void tc_teardown(TileCommon &c, uint32_t ncols, uint32_t phase) {
    if (c.abort) tc::mbar_wait_bounded(&c.mbar, phase ^ 1u, 1u << 22);  // let an MMA in flight finish
    cp_async_wait_all();
    tc::fence_before_sync();
    __syncthreads();
    if (threadIdx.x < 32) tc::tmem_dealloc(c.tmem, ncols);
}

// Waits for the MMAs of the current item.  On a timeout the abort flag is set; the
// thread goes on to the item's last barrier, after which every thread sees the flag
// and leaves (a barrier here would only carry the flag: each thread waits by itself).
__device__ __forceinline__ void tc_wait(TileCommon &c, uint32_t phase, int *status) {
    if (!tc::mbar_wait_bounded(&c.mbar, phase, 1u << 24)) {
        atomicOr(status, kStatTimeout);
        c.abort = 1;
    }
    tc::fence_after_sync();
}

// The pair loop of a tile: item it + 1 is copied while item it is processed.  Item
// it is visible to all threads and every thread is done with the other slot:
// first_pair ends with a barrier.
template <class Buf>
__device__ __forceinline__ int next_pair(TileCommon &cm, Buf *pb, const MixedArgs &A, int64_t it, int64_t it0,
                                         int64_t it1, uint64_t &nxt, bool with_coef) {
    const int cur = (int)((it - it0) & 1);
    if (it + 1 < it1) {
        fetch_pair(pb[cur ^ 1].hdr_, cm.ii[cur ^ 1], A, it + 1, nxt, with_coef);
        if (it + 2 < it1) nxt = A.items[it + 2];
    }
    return cur;
}
template <class Buf>
__device__ __forceinline__ void first_pair(TileCommon &cm, Buf *pb, const MixedArgs &A, int64_t it0, int64_t it1,
                                           uint64_t &nxt, bool with_coef) {
    if (it0 < it1) fetch_pair(pb[0].hdr_, cm.ii[0], A, it0, A.items[it0], with_coef);
    if (it0 + 1 < it1) nxt = A.items[it0 + 1];
    cp_async_wait_all();
    __syncthreads();
}

// Stage 1 of collocate: Cxy[z][(b,a)] = sum_g c'[g][b][a] Z[g][z]; one (b, a) and two
// z per thread (packed float-float), two partial sums over even and odd g; the
// packed index of (g, b, a) is zs[g] - b g + k0.  Rows b of Cxy are padded to an even
// number of a (the padding gets zeros), so that stage 2 reads its pairs of a as
// 16-byte entries {hi(a), hi(a+1), lo(a), lo(a+1)}.
__device__ __forceinline__ void stage1_cxy(SmemColl &sm, int L, int lp, const TileShape &sh) {
    const int *zs = c_zs[lp];
    const int npad = 2 * (L >> 1) * ((L >> 1) + 1) + (L & 1) * (L + 1);  // cxy_pad_row(L, L)
    for (int t = (int)threadIdx.x - 32; t < (npad << (sh.lz - 1)); t += NTHR - 32) {
        const int zz = 2 * (t & ((sh.TZ >> 1) - 1));
        const uint32_t de = sm.st1[lp][t >> (sh.lz - 1)];
        const int b = de & 15, a = de >> 4, n = lp - a - b;
        const int q = b * L - (b * (b - 1)) / 2 + ((b + (L & 1)) >> 1) + a;  // cxy_pad_row(L, b) + a
        const ff *c = sm.rc + (b * (lp + 1) - (b * (b - 1)) / 2 + a);
        ff2 s0 = {f2(0.0f), f2(0.0f)}, s1 = s0;
        auto zpair = [&](int g) {
            return ff2n{*reinterpret_cast<const float2 *>(&sm.Zh[g][zz]), *reinterpret_cast<const float2 *>(&sm.Znh[g][zz]),
                        *reinterpret_cast<const float2 *>(&sm.Znl[g][zz])};
        };
        int g = 0, bg = 0;
#pragma unroll 1
        for (; g + 1 <= n; g += 2, bg += 2 * b) {
            s0 = ff2_fma(ff2_dup(c[zs[g] - bg]), zpair(g), s0);
            s1 = ff2_fma(ff2_dup(c[zs[g + 1] - bg - b]), zpair(g + 1), s1);
        }
        if (g <= n) s0 = ff2_fma(ff2_dup(c[zs[g] - bg]), zpair(g), s0);
        s0 = ff2_add(s0, s1);
        float *o = reinterpret_cast<float *>(&sm.Cxy[zz][q >> 1]) + (q & 1);
        o[0] = s0.hi.x;
        o[2] = s0.lo.x;
        o += 4 * kCxyRow;
        o[0] = s0.hi.y;
        o[2] = s0.lo.y;
    }
}

// Stage 2 of collocate for this thread's row (z, y): Cx[a] = sum_b Cxy[z][b][a] Y[b][y],
// two a per instruction, then the row's A slices (K slots below kw rewritten);
// returns the row exponent.  b outer, the pairs of a unrolled inside (uniform exit at
// the row's end), so that Y is read once per b; each sum renormalised once at the end.
__device__ __forceinline__ int stage2_row(SmemColl &sm, int L, int lp, int z, int y, bool live,
                                          int kw, int m) {
    ff2 cx[kNPair];
#pragma unroll
    for (int i = 0; i < kNPair; i++) cx[i] = ff2{f2(0.0f), f2(0.0f)};
    float mx = 0.0f;
    if (live) {
        const float4 *crow = sm.Cxy[z];
#pragma unroll 1
        for (int b = 0; b <= lp; b++) {
            const ff2n yb = ff2n_dup(sm.Y[b][y]);
#pragma unroll
            for (int i = 0; i < kNPair; i++) {
                if (2 * i > lp - b) break;
                const float4 c = crow[i];
                ff2_acc_lazy(cx[i], ff2{make_float2(c.x, c.y), make_float2(c.z, c.w)}, yb);
            }
            crow += (L - b + 1) >> 1;
        }
#pragma unroll
        for (int i = 0; i < kNPair; i++) {
            cx[i] = fast_two_sum2(cx[i].hi, cx[i].lo);
            mx = fmaxf(mx, fmaxf(fabsf(cx[i].hi.x), fabsf(cx[i].hi.y)));  // entries a > lp are zero
        }
    }
    const int em = exp_of(mx);
    const float sc = em == kZeroExp ? 0.0f : pow2i(SLB - em);
    // entries a > lp of cx are zero; K slots that may hold an earlier pair's values are rewritten
    slice_row16(cx, sc, kw, L, sm.A[0], MROWS * KP, m);
    return em;
}

// ---------------------------------------------------------------------------
// kGeneral: tiles of general-cell levels.  The tables, stages and slices are the
// same in t_d = (index_d - gp_d) |v_d|; the row ranges come from the quadratic
// rule, and every point's value is multiplied by the cross factor
// E = exp(-2 zetp (c01 t0 t1 + c02 t0 t2 + c12 t1 t2)) of the Gaussian
// (exp(-zetp |r|^2) = exp(-zetp (t0^2 + t1^2 + t2^2)) E).  Along a row E(x) is
// exp(alpha + beta t0(x)): one exp at the row's first cube point, then E(x+1) =
// E(x) q, q = exp(beta |v0|), over the row's cube points only (so no intermediate
// leaves the range of the factor inside the cube).
template <bool kGeneral>
__global__ void __launch_bounds__(NTHR, 4) k_collocate_tiled(MixedArgs A) {
    extern __shared__ __align__(128) unsigned char smraw[];
    SmemColl &sm = *reinterpret_cast<SmemColl *>(smraw);
    TileCommon &cm = sm.c;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int m = tid;
    constexpr uint32_t kCols = 128;  // diagonals D2..D5: 32 columns each
    tc_setup(cm, kCols);
    const uint32_t tbase = cm.tmem + ((uint32_t)(warp * 32) << 16);
    uint32_t phase = 0;
    int kprev = KP;  // K slots of A and B that the previous pair wrote (uninitialised at first: all)
    for (int t = tid; t < kNPow * 2 * kCxyRow; t += NTHR) (&sm.st1[0][0])[t] = (&d_order.st1[0][0])[t];
    for (int t = tid; t < kNPow * kNPow; t += NTHR) sm.bin[t / kNPow][t % kNPow] = c_binom[t / kNPow][t % kNPow];
    for (;;) {
        if (tid == 0) cm.tile = atomicAdd(A.queue, 1);
        __syncthreads();
        const int tile = cm.tile;
        if (tile >= A.ntiles || cm.abort) break;
        const TileDesc td = A.tiles[tile];
        const LevelDev &lv = A.levels[td.level];
        const TileShape sh(td.lz);
        const int TY = sh.TY, TZ = sh.TZ;
        // a warp's 32 rows: 8 y x 4 z, so that more warps (and chunks) lie wholly outside a sphere
        const int wy = TY >> 3, y = (warp & (wy - 1)) * 8 + (m & 7), z = (warp / wy) * 4 + ((m >> 3) & 3);
        float2 acc_hi[TX / 2];  // pairs of x; the low parts live in shared memory (registers for 4 CTAs per SM)
        float *acc_lo = sm.acc_lo[m];
#pragma unroll
        for (int x = 0; x < TX; x++) acc_lo[x] = 0.0f;
#pragma unroll
        for (int x = 0; x < TX / 2; x++) acc_hi[x] = f2(0.0f);
        const TileExt ext = {min(TX, lv.ngrid[0] - td.t[0] * TX), min(TY, lv.ngrid[1] - td.t[1] * TY),
                             min(TZ, lv.ngrid[2] - td.t[2] * TZ)};
        const bool row_ok = z < ext.z && y < ext.y;
        const int64_t it0 = A.start[2 * tile], it1 = A.start[2 * tile + 1];
        uint64_t nxt = 0;
        first_pair(cm, sm.pb, A, it0, it1, nxt, true);
        for (int64_t it = it0; it < it1; it++) {
            const int cur = (int)((it - it0) & 1);
            if constexpr (!kGeneral) next_pair(cm, sm.pb, A, it, it0, it1, nxt, true);
            const PairBuf &pb = sm.pb[cur];
            const TPair &P = pb.p;
            const int L = P.L, lp = P.lp;
            const ImgState &Q = cm.ii[cur].im;
            {
                // warp 0: X column (lane x) and its B slices, scaled by 2^(SLB - fx); warp 1:
                // Y and Z tables; warps 2-3: re-expansion of the coefficients
                if (warp < 2) {
#pragma unroll 1
                    for (int ent = tid & 31; ent < (warp == 0 ? TX : TY + TZ); ent += 32) {
                        const TabEntry te = tab_entry(P, Q, ext, sh, cm.exptab, warp, ent);
                        if (warp == 0) {
                            // the powers of u, two per step, in rolled loops: once for their
                            // maximum, once to be sliced (K slots beyond L may hold an earlier
                            // pair's slices: rewritten as zeros)
                            const ff u = ff_mul_f(P.h[0], ldexpf((float)(ent - Q.ic), -Q.sb));
                            const ff2n u2 = ff2n_dup(ff_mul(u, u));
                            ff2 xa = te.in ? ff2_pair(te.e, ff_mul(te.e, u)) : ff2{f2(0.0f), f2(0.0f)};
                            float mx = 0.0f;
                            ff2 xb = xa;
#pragma unroll 1
                            for (int a = 0; a < L; a += 2) {
                                mx = fmaxf(mx, a + 1 < L ? fmaxf(fabsf(xb.hi.x), fabsf(xb.hi.y)) : fabsf(xb.hi.x));
                                xb = ff2_mul(xb, u2);
                            }
                            const int e = exp_of(mx);
                            sm.cs[cur][tid] = e == kZeroExp ? 0.0f : pow2i(e);
                            const float sc = e == kZeroExp ? 0.0f : pow2i(SLB - e);
                            uint32_t *bp = reinterpret_cast<uint32_t *>(sm.B[0]) + (tid >> 3) * 64 + (tid & 7) * 4;
                            const int kw = (max(L, kprev) + 7) & ~7;
#pragma unroll 1
                            for (int a = 0; a < kw; a += 2) {
                                if (a >= L) xa = ff2{f2(0.0f), f2(0.0f)};
                                if (a + 1 >= L) xa.hi.y = xa.lo.y = 0.0f;
                                float2 sl[NSL];
                                slice_scaled2(xa, f2(sc), sl);
#pragma unroll
                                for (int q = 0; q < NSL; q++)
                                    bp[q * (TX * KP / 2) + (a >> 3) * 32 + ((a & 7) >> 1)] = pack_halves(sl[q]);
                                xa = ff2_mul(xa, u2);
                            }
                        } else {
                            yz_fill(sm, P, te, 0);
                        }
                    }
                } else {
                    recentre_x(pb, Q.tc, Q.sb, sm.rc, sm.bin, 64, NTHR - 64);
                }
                // stage 1 needs the z table and the re-expansion, not the x slices: warps 1-3
                // go on to it while warp 0 still slices
                if (warp > 0) {
                    asm volatile("bar.sync 2, 96;" ::: "memory");
                    stage1_cxy(sm, L, lp, sh);
                }
                __syncthreads();
                if (cm.abort) break;  // uniform: set before this barrier or after the next one
                // (general cell: every warp is done with the previous item's record here)
                if constexpr (kGeneral) next_pair(cm, sm.pb, A, it, it0, it1, nxt, true);
                // stage 2 (this thread's row, all a at once) + culling + A slices
                int x0, x1;
                if constexpr (kGeneral)
                    general_row_range(lv, A.glv[td.level], P, Q, Q.o[2] + z, Q.o[1] + y, row_ok, x0,
                                      x1);
                else
                    row_range(P, Q, A.table, Q.o[2] + z, Q.o[1] + y, row_ok, x0, x1);
                const int em = stage2_row(sm, L, lp, z, y, x0 <= x1, max(L, kprev), m);
                // stage 3 on the tensor cores: D_s = sum_{i+j=s} A_i B_j^T
                // What follows reads none of the tables, and the record only on general cells:
                // the next item's record, waited for here, and its tables may come in as the
                // warps finish their readout, and no barrier ends the item (64.2 -> 62.4 ms,
                // 100k pairs, 256^3).
                cp_async_wait_all();
                tc::fence_async_smem();
                tc::fence_before_sync();
                __syncthreads();
                if (tid == 0) {
                    tc::fence_after_sync();
                    // diagonal s = i + j into TMEM columns [32 s, 32 s + 32): the planes of B lie
                    // one after the other along N, so A_i times B_0 .. B_{3-i} is one MMA of
                    // N = 32 (4 - i) whose columns start at 32 i (4 MMAs instead of 10)
                    const uint64_t ad = tc::desc_kmajor(sm.A[0], 128, 256), bd = tc::desc_kmajor(sm.B[0], 128, 256);
#pragma unroll
                    for (int i = 0; i < NSL; i++)
                        tc::mma_f16(cm.tmem + 32 * i, ad + (uint64_t)(i * (int)sizeof(sm.A[0]) >> 4), bd,
                                    tc::idesc_f16_f32(MROWS, TX * (NSL - i)), i > 0);
                    tc::mma_commit(&cm.mbar);
                }
                tc_wait(cm, phase, A.status);
                phase ^= 1u;
                kprev = L;
                // cross factor of the general cell along this row, two x at a time
                ff2 ecur = {f2(1.0f), f2(0.0f)};
                ff2n eq = {};
                if constexpr (kGeneral) {
                    if (x0 <= x1) cross_factor_row(A.glv[td.level], P, Q, cm.exptab, z, y, x0, ecur, eq);
                }
                // tcgen05.ld is warp-collective: chunk decisions are made per warp
                if (__any_sync(0xffffffffu, x0 <= x1)) {
                    const float rs = pow2i(max(em - 2 * SLB, -126));
                    // bits x0..x1 of the row: the points of this pair's sphere on the row
                    const uint32_t rmask =
                        x0 > x1 ? 0u : (uint32_t)(((2ull << x1) - 1ull) & ~((1ull << x0) - 1ull));
                    // kCh chunks of 8 x per iteration; acc_hi[0 .. 8 kCh) always holds the current
                    // chunks' sums, rotated by 8 kCh after each iteration (TX / (8 kCh)
                    // rotations restore the order).  All four chunks in line need no
                    // rotation, and with packed arithmetic the code still fits the
                    // instruction cache: 73.2, 71.5 and 66.8 ms with 1, 2 and 4 chunks (100k
                    // pairs, 256^3).  The general-cell body, longer by the cross factor, keeps
                    // one chunk: 7.36, 7.95 and 8.72 ms (8000 pairs, 128^3).
                    constexpr int kCh = kGeneral ? 1 : 4;
#pragma unroll 1
                    for (int c2 = 0; c2 < TX / (8 * kCh); c2++) {
#pragma unroll
                        for (int hh = 0; hh < kCh; hh++) {
                            const int c = kCh * c2 + hh;
                            const uint32_t mc = rmask >> (8 * c);
                            if (__any_sync(0xffffffffu, (mc & 0xFFu) != 0u)) {
                                uint32_t r2[8], r3[8], r4[8], r5[8];
                                const float4 csa = reinterpret_cast<const float4 *>(sm.cs[cur])[2 * c];
                                const float4 csb = reinterpret_cast<const float4 *>(sm.cs[cur])[2 * c + 1];
                                const float2 csv[4] = {{csa.x, csa.y}, {csa.z, csa.w}, {csb.x, csb.y}, {csb.z, csb.w}};
                                tc::tmem_ld8(tbase + 8 * c, r2);
                                tc::tmem_ld8(tbase + 32 + 8 * c, r3);
                                tc::tmem_ld8(tbase + 64 + 8 * c, r4);
                                tc::tmem_ld8(tbase + 96 + 8 * c, r5);
                                float4 *const lop = reinterpret_cast<float4 *>(acc_lo) + 2 * c;
                                const float4 loa = lop[0], lob = lop[1];
                                float2 lov[4] = {{loa.x, loa.y}, {loa.z, loa.w}, {lob.x, lob.y}, {lob.z, lob.w}};
                                tc::tmem_wait_ld32(r2, r3, r4, r5);
#pragma unroll
                                for (int i = 0; i < 4; i++) {  // two x per instruction, selects instead of branches
                                    const bool in0 = (mc >> (2 * i)) & 1u, in1 = (mc >> (2 * i + 1)) & 1u;
                                    auto two = [&](const uint32_t *r) {
                                        return make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
                                    };
                                    // value = scl * (D2 + D3 2^-10 + D4 2^-20 + D5 2^-30) as hi + lo with
                                    // lo the exact remainder (fast two-sum), then an exact two-sum into
                                    // acc_hi: acc_lo then only gathers rounding errors and remainders,
                                    // so it stays ~2^-24 below acc_hi however many pairs a point sees
                                    const float2 d2 = two(r2);
                                    const float2 corr =
                                        f2_fma(two(r5), f2(9.313225746154785e-10f),
                                               f2_fma(two(r4), f2(9.5367431640625e-07f), f2_mul(two(r3), f2(0.0009765625f))));
                                    float2 scl = f2_mul(f2(rs), csv[i]);
                                    const float2 h0 = f2_add(d2, corr);
                                    float2 hi = f2_mul(h0, scl);
                                    float2 rem = f2_sub(corr, f2_sub(h0, d2));  // lo = rem scl exactly
                                    if constexpr (kGeneral) {
                                        const int x = 8 * c + 2 * i;
                                        if (x > x0 && x <= x1) ecur = next_cross(ecur, eq);  // E on the row's cube points
                                        const ff2 v = ff2_mul(ff2{hi, f2_mul(rem, scl)}, ff2n_of(ecur));
                                        hi = v.hi;
                                        rem = v.lo;
                                        scl = f2(1.0f);
                                    }
                                    float2 &ah = acc_hi[4 * hh + i];
                                    const float2 sv = f2_add(ah, hi);
                                    const float2 bb = f2_sub(sv, ah);
                                    const float2 err = f2_add(f2_sub(ah, f2_sub(sv, bb)), f2_sub(hi, bb));
                                    const float2 lo = f2_add(lov[i], f2_fma(rem, scl, err));
                                    ah = make_float2(in0 ? sv.x : ah.x, in1 ? sv.y : ah.y);
                                    lov[i] = make_float2(in0 ? lo.x : lov[i].x, in1 ? lo.y : lov[i].y);
                                }
                                lop[0] = make_float4(lov[0].x, lov[0].y, lov[1].x, lov[1].y);
                                lop[1] = make_float4(lov[2].x, lov[2].y, lov[3].x, lov[3].y);
                            }
                        }
                        float2 tr[4 * kCh];
#pragma unroll
                        for (int i = 0; i < 4 * kCh; i++) tr[i] = acc_hi[i];
#pragma unroll
                        for (int i = 0; i < TX / 2 - 4 * kCh; i++) acc_hi[i] = acc_hi[i + 4 * kCh];
#pragma unroll
                        for (int i = 0; i < 4 * kCh; i++) acc_hi[TX / 2 - 4 * kCh + i] = tr[i];
                    }
                }
            }
        }
        __syncthreads();
        if (cm.abort) break;
        // flush: grid += tile sum (FP64)
        if (row_ok) {
            double *grid = A.grids.p[td.level];
            const int64_t row = ((int64_t)(td.t[2] * TZ + z) * lv.ngrid[1] + (td.t[1] * TY + y)) * lv.ngrid[0] +
                                td.t[0] * TX;
            // 8 points per iteration, acc_hi rotated by 8 after each (compact code); all eight
            // loads first (left to the compiler, one build loaded, added and stored point by
            // point: 1000 pairs on 256^3, 20 items a unit, 1.56 against 0.69 ms)
            const bool split = td.flags & kUnitSplit;  // other work units add to the same tile
#pragma unroll 1
            for (int c = 0; c < TX / 8; c++) {
                double g8[8];
#pragma unroll
                for (int i = 0; i < 8; i++) g8[i] = split || 8 * c + i >= ext.x ? 0.0 : grid[row + 8 * c + i];
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const int x = 8 * c + i;
                    if (x >= ext.x) continue;
                    const double v = (double)(i & 1 ? acc_hi[i / 2].y : acc_hi[i / 2].x) + (double)acc_lo[x];
                    if (split) atomicAdd(grid + row + x, v);
                    else grid[row + x] = g8[i] + v;
                }
#pragma unroll
                for (int i = 0; i < TX / 2 - 4; i++) acc_hi[i] = acc_hi[i + 4];
            }
        }
        __syncthreads();
    }
    tc_teardown(cm, kCols, phase);
}

// s += four products a b, the even and the odd ones in the two halves of s
__device__ __forceinline__ void acc_four(ff2 &s, float4 ah, float4 al, float4 bh, float4 bnh, float4 bnl) {
    ff2_acc_lazy(s, ff2{make_float2(ah.x, ah.y), make_float2(al.x, al.y)},
                 ff2n{make_float2(bh.x, bh.y), make_float2(bnh.x, bnh.y), make_float2(bnl.x, bnl.y)});
    ff2_acc_lazy(s, ff2{make_float2(ah.z, ah.w), make_float2(al.z, al.w)},
                 ff2n{make_float2(bh.z, bh.w), make_float2(bnh.z, bnh.w), make_float2(bnl.z, bnl.w)});
}

// Stage 1 transposed: the moments W[g][b][a] += sum_z T[z][(b,a)] Z[g][z]
// of an item of degree lp, by 96 threads (t0 of 96).  T lies in the columns of S that a
// warp was done with: pass p of its (b,a) in row lp - p (see stage 2 transposed).  It is
// a serial chain of loads and sums; run between barriers of its own it took 3.5 of 56 ms
// of 100k pairs on 256^3, beside the next item's tables it takes none of the item's path.
template <class Smem>
__device__ __forceinline__ void add_moments(const Smem &sm, double *mom, int lp, int zbuf, const TileShape &sh, int t0) {
    const int nc = ncoef(lp), lzw = 5 - sh.ly;
    for (int t = t0; t < nc; t += 96) {
        const uint32_t de = __ldg(&d_decode.e[d_decode_at(lp) + t]);  // (g, b, a) of packed index t
        const int g = de & 15, pi = de >> 16;
        const int p = pi >> (5 - lzw), col = (pi << lzw) & 31;
        const float *th = sm.st.Sh[lp - p] + col, *tl = sm.st.Sl[lp - p] + col;
        ff2 s2 = {f2(0.0f), f2(0.0f)};
#pragma unroll 1
        for (int z4 = 0; z4 < sh.TZ; z4 += 4) {
            float4 h, l;
            if (lzw) {  // two z per warp: (z, z + 1) in one column pair of warp z / 2
                const float2 h0 = *reinterpret_cast<const float2 *>(th + 16 * z4),
                             h1 = *reinterpret_cast<const float2 *>(th + 16 * z4 + 32);
                const float2 l0 = *reinterpret_cast<const float2 *>(tl + 16 * z4),
                             l1 = *reinterpret_cast<const float2 *>(tl + 16 * z4 + 32);
                h = make_float4(h0.x, h0.y, h1.x, h1.y);
                l = make_float4(l0.x, l0.y, l1.x, l1.y);
            } else {  // one z per warp
                h = make_float4(th[32 * z4], th[32 * z4 + 32], th[32 * z4 + 64], th[32 * z4 + 96]);
                l = make_float4(tl[32 * z4], tl[32 * z4 + 32], tl[32 * z4 + 64], tl[32 * z4 + 96]);
            }
            const float4 zh = *reinterpret_cast<const float4 *>(&sm.Zh[zbuf][g][z4]);
            acc_four(s2, h, l, zh, make_float4(-zh.x, -zh.y, -zh.z, -zh.w),
                     *reinterpret_cast<const float4 *>(&sm.Znl[zbuf][g][z4]));
        }
        const ff s = ff_add(ff{s2.hi.x, s2.lo.x}, ff{s2.hi.y, s2.lo.y});
        if (s.hi != 0.0f) atomicAdd(mom + t, ff_to_double_bits(s));
    }
}

// kGeneral: tiles of general-cell levels; the A operand holds the slices of
// V(x) E(x) (E the cross factor of the Gaussian along the row), one row per
// thread, with its own exponent per row and image.
template <bool kGeneral>
__global__ void __launch_bounds__(NTHR, 4) k_integrate_tiled(MixedArgs A) {
    extern __shared__ __align__(128) unsigned char smraw[];
    SmemInt &sm = *reinterpret_cast<SmemInt *>(smraw);
    uint4 *const vslot = A.vslot + (size_t)blockIdx.x * kVSlot16;
    TileCommon &cm = sm.c;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int m = tid;
    constexpr uint32_t kCols = 128;  // D2 (two K halves), D3, D4, D5: 16 columns each
    tc_setup(cm, kCols);
    const uint32_t tbase = cm.tmem + ((uint32_t)(warp * 32) << 16);
    uint32_t phase = 0;
    // B rows alpha >= L are never written: start them finite (zero)
    for (int t = tid; t < (int)(sizeof(sm.B) / sizeof(uint4)); t += NTHR)
        reinterpret_cast<uint4 *>(sm.B)[t] = make_uint4(0u, 0u, 0u, 0u);
    for (;;) {
        if (tid == 0) cm.tile = atomicAdd(A.queue, 1);
        __syncthreads();
        const int tile = cm.tile;
        if (tile >= A.ntiles || cm.abort) break;
        const TileDesc td = A.tiles[tile];
        const LevelDev &lv = A.levels[td.level];
        const TileShape sh(td.lz);
        const int TY = sh.TY, TZ = sh.TZ, z = m >> sh.ly, y = m & (TY - 1);
        const TileExt ext = {min(TX, lv.ngrid[0] - td.t[0] * TX), min(TY, lv.ngrid[1] - td.t[1] * TY),
                             min(TZ, lv.ngrid[2] - td.t[2] * TZ)};
        const bool row_ok = z < ext.z && y < ext.y;
        // this thread's V row, sliced once per tile (row exponent vm), into A and the slot
        int vm;
        {
            const double *grid = A.grids.p[td.level];
            const int64_t row = ((int64_t)(td.t[2] * TZ + z) * lv.ngrid[1] + (td.t[1] * TY + y)) * lv.ngrid[0] +
                                td.t[0] * TX;
            // compact loops (once per unit): the row as float-float and its maximum, then
            // 16-byte chunks of 8 x; 8 loads in flight (one at a time, their latency was a
            // tenth of a 16-item unit).  Between the two the row lies where its slices will
            // (as many bytes), and the split is done on the integer pipe (read twice and split
            // by conversions, 17 cycles a warp each: 1000 pairs on 64^3, units of 31 items, 261
            // against 240 us; three levels, units of 60, 3.86 against 3.80 ms).
            float mx = 0.0f;
#pragma unroll 1
            for (int c = 0; c < TX / 8; c++) {
                const int o16 = (m >> 3) * 16 + (c & 1) * 8 + (m & 7);  // offset of (m, 8 c) / 16
                double v8[8];
#pragma unroll
                for (int i = 0; i < 8; i++) v8[i] = (row_ok && 8 * c + i < ext.x) ? grid[row + 8 * c + i] : 0.0;
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    ff v0, v1;
                    if constexpr (kGeneral) {  // (shorter code counts for more: 6.76 against 6.83 ms)
                        v0 = ff_from_double(v8[2 * i]);
                        v1 = ff_from_double(v8[2 * i + 1]);
                    } else {
                        const bool in0 = row_ok && 8 * c + 2 * i < ext.x, in1 = row_ok && 8 * c + 2 * i + 1 < ext.x;
                        v0 = in0 ? ff_from_double_bits(v8[2 * i]) : ff{0.0f, 0.0f};
                        v1 = in1 ? ff_from_double_bits(v8[2 * i + 1]) : ff{0.0f, 0.0f};
                    }
                    const float4 v = make_float4(v0.hi, v0.lo, v1.hi, v1.lo);
                    if constexpr (kGeneral) reinterpret_cast<float4 *>(vslot)[(4 * c + i) * MROWS + m] = v;
                    else reinterpret_cast<float4 *>(sm.A[c >> 1][i])[o16] = v;
                    mx = fmaxf(mx, fmaxf(fabsf(v0.hi), fabsf(v1.hi)));
                }
            }
            vm = exp_of(mx);
            const float sc = vm == kZeroExp ? 0.0f : pow2i(SLB - vm);
#pragma unroll 1
            for (int c = 0; c < TX / 8 && !kGeneral; c++) {  // 8 x per 16-byte chunk of the UMMA layout
                const int o16 = (m >> 3) * 16 + (c & 1) * 8 + (m & 7);
                uint32_t w[NSL][4];
                static_assert(NSL == 4, "8 float-float values fill the chunks of their slices");
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const float4 v = reinterpret_cast<const float4 *>(sm.A[c >> 1][i])[o16];
                    float2 sl[NSL];
                    slice_scaled2(ff2{make_float2(v.x, v.z), make_float2(v.y, v.w)}, f2(sc), sl);
#pragma unroll
                    for (int q = 0; q < NSL; q++) w[q][i] = pack_halves(sl[q]);
                }
#pragma unroll
                for (int q = 0; q < NSL; q++) {
                    const uint4 val = make_uint4(w[q][0], w[q][1], w[q][2], w[q][3]);
                    vslot[((c >> 1) * NSL + q) * (MROWS * KP / 8) + o16] = val;
                    reinterpret_cast<uint4 *>(sm.A[c >> 1][q])[o16] = val;
                }
            }
            if constexpr (!kGeneral) __threadfence();  // the slot's rows are read back by cp.async
        }
        const int64_t it0 = A.start[2 * tile], it1 = A.start[2 * tile + 1];
        uint64_t nxt = 0;
        first_pair(cm, sm.pb, A, it0, it1, nxt, false);
        uint32_t M = 0, have = ~0u;  // this row's points in the current item, and those its A row holds
        if constexpr (!kGeneral) {
            if (it0 < it1) M = row_mask(sm.pb[0].p, cm.ii[0].im, A.table, z, y, row_ok);
            sm.mask[m] = M;
            sm.todo[m] = chunks_to_mask(M, have);
            __syncthreads();
        }
        // the item whose moments are still to be added (by warps 1-3, while warp 0 makes the
        // next item's B): its degree and moments
        int lp_done = -1;
        double *mom_done = nullptr;
        for (int64_t it = it0; it < it1; it++) {
            const int cur = next_pair(cm, sm.pb, A, it, it0, it1, nxt, false);
            const TPair &P = sm.pb[cur].p;
            const int L = P.L, lp = P.lp;
            const int npair = (L * (L + 1)) / 2;
            const int64_t moff = P.coef_off;
            const ImgState &Q = cm.ii[cur].im;
            {
                int x0 = 1, x1 = 0, vrow = vm;
                if constexpr (kGeneral) {  // every thread: its row's cube x range and its A row
                    general_row_range(lv, A.glv[td.level], P, Q, Q.o[2] + z, Q.o[1] + y, row_ok, x0, x1);
                    vrow = general_a_row(sm, vslot, A.glv[td.level], P, Q, sh, m, x0, x1);
                }
                // Code size counts: four CTAs per SM at different points of the loop share the
                // instruction caches, and the general-cell kernel, which has the row rule
                // and the cross factor as well, lost a fifth of its issue slots to fetches.
                // It has one copy of the table code (7.13 ms with the compact B loop below,
                // 7.93 without either, 6.86 with stage 2 transposed rolled as well); the
                // orthorhombic one is faster with a copy per warp (53.0 against 53.7 ms,
                // 100k pairs, 256^3), with stage 2 unrolled by 4 (53.0 against 53.4).
                TabEntry te0;
                if constexpr (kGeneral) {
                    if (warp < 2) {
#pragma unroll 1
                        for (int ent = tid & 31; ent < (warp == 0 ? TX : TY + TZ); ent += 32) {
                            te0 = tab_entry(P, Q, ext, sh, cm.exptab, warp, ent);
                            if (warp == 1) yz_fill(sm, P, te0, cur);
                        }
                    }
                }
                if (warp == 0) {
                    // B: row alpha = X[alpha][x] over x (lane x), two alpha at a time, scaled by
                    // 2^(SLB - g[alpha]) (maximum over the warp); rows alpha >= L are left as
                    // they are (their output columns are not read).  The powers are formed as
                    // the loop goes (unrolled over a table in registers: 53.5 against 53.0 ms).
                    if constexpr (!kGeneral) te0 = tab_entry(P, Q, ext, sh, cm.exptab, 0, tid);
                    if (!te0.in) te0.e = te0.t = ff{0.0f, 0.0f};
                    ff2 xa = ff2_pair(te0.e, ff_mul(te0.e, te0.t));  // alpha, alpha + 1
                    const ff2n u2 = ff2n_dup(ff_mul(te0.t, te0.t));
#pragma unroll 1
                    for (int a = 0; a < L; a += 2) {
                        if (a + 1 >= L) xa.hi.y = xa.lo.y = 0.0f;
                        // per-alpha maximum over x: one warp reduction (the bit patterns of
                        // non-negative floats order as their values)
                        float sc[2];
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            const float mxb =
                                __uint_as_float(__reduce_max_sync(
                                    0xffffffffu, __float_as_uint(fabsf(h ? xa.hi.y : xa.hi.x))));
                            const int e = exp_of(mxb);
                            if (tid == a + h) sm.gsc[a + h] = e == kZeroExp ? 0.0f : pow2i(e - SLB);
                            sc[h] = e == kZeroExp ? 0.0f : pow2i(SLB - e);
                        }
                        float2 sl[NSL];
                        slice_scaled2(xa, make_float2(sc[0], sc[1]), sl);
                        unsigned char *const bp = sm.B + (tid >> 4) * kBHalf + b_off(a, tid & 15);
#pragma unroll
                        for (int q = 0; q < NSL; q++) {
                            const uint32_t w = pack_halves(sl[q]);
                            *reinterpret_cast<uint16_t *>(bp + q * kBPlane) = (uint16_t)w;
                            *reinterpret_cast<uint16_t *>(bp + q * kBPlane + 16) = (uint16_t)(w >> 16);
                        }
                        xa = ff2_mul(xa, u2);
                    }
                } else if (!kGeneral && warp == 1) {
#pragma unroll 1
                    for (int ent = tid - 32; ent < TY + TZ; ent += 32)
                        yz_fill(sm, P, tab_entry(P, Q, ext, sh, cm.exptab, 1, ent), cur);
                    if (lp_done >= 0) add_moments(sm, mom_done, lp_done, cur ^ 1, sh, tid + 32);
                } else if constexpr (!kGeneral) {
                    if (lp_done >= 0) add_moments(sm, mom_done, lp_done, cur ^ 1, sh, tid - 64);
                    mask_a_row(sm, tid - 64, sm.mask[tid - 64], sm.todo[tid - 64]);
                    mask_a_row(sm, tid, sm.mask[tid], sm.todo[tid]);
                }
                if constexpr (kGeneral) {
                    if (warp >= 1 && lp_done >= 0)
                        add_moments(sm, mom_done, lp_done, cur ^ 1, sh, warp == 1 ? tid + 32 : tid - 64);
                }
                cp_async_wait_all();  // the next item's record, read after this barrier
                tc::fence_async_smem();
                tc::fence_before_sync();
                __syncthreads();
                if (tid == 0) {
                    tc::fence_after_sync();
                    // as in collocate, A_i of K half h times the planes B_0 .. B_{3-i} in one MMA
                    // of N = 16 (4 - i), diagonal s into columns [16 + 16 s, 32 + 16 s); D2 of the
                    // second half apart, in columns [0, 16) (exact: 16 products each): 9 MMAs
                    // instead of 20
                    const uint64_t ad = tc::desc_kmajor(sm.A[0][0], 128, 256), bd = tc::desc_kmajor(sm.B, kBLbo, kBSbo);
                    constexpr uint64_t kA = sizeof(sm.A[0][0]) >> 4, kB1 = kBHalf >> 4, kBP = kBPlane >> 4;
#pragma unroll
                    for (int i = 0; i < NSL; i++)
                        tc::mma_f16(cm.tmem + 16 + 16 * i, ad + kA * i, bd, tc::idesc_f16_f32(MROWS, KP * (NSL - i)), i > 0);
                    tc::mma_f16(cm.tmem, ad + kA * NSL, bd + kB1, tc::idesc_f16_f32(MROWS, KP), 0);
                    tc::mma_f16(cm.tmem + 32, ad + kA * NSL, bd + kB1 + kBP, tc::idesc_f16_f32(MROWS, KP * (NSL - 1)), 1);
#pragma unroll
                    for (int i = 1; i < NSL; i++)
                        tc::mma_f16(cm.tmem + 16 + 16 * i, ad + kA * (NSL + i), bd + kB1,
                                    tc::idesc_f16_f32(MROWS, KP * (NSL - i)), 1);
                    tc::mma_commit(&cm.mbar);
                }
                // while the MMAs run: the next item's range of this row (after them: 51.9 against
                // 51.1 ms, 100k pairs on 256^3; in collocate, whose code grows by it, 59.9 against
                // 58.7 the other way round)
                uint32_t Mn = 0u;
                if constexpr (!kGeneral)
                    if (it + 1 < it1) Mn = row_mask(sm.pb[cur ^ 1].p, cm.ii[cur ^ 1].im, A.table, z, y, row_ok);
                tc_wait(cm, phase, A.status);
                phase ^= 1u;
                const bool live = kGeneral ? x0 <= x1 : M != 0u;  // other rows give zeros
                if constexpr (!kGeneral) {
                    // what A lacks of it
                    if (M != 0u) have = M;
                    M = Mn;
                    if (it + 1 < it1) {
                        have = restore_a_row(sm, vslot, m, M, have);
                        sm.mask[m] = M;
                        sm.todo[m] = chunks_to_mask(M, have);
                    }
                }
                // A warp whose rows all lie outside has only zeros to hand on (3.95 -> 3.86 ms on
                // the three-level workload, 53.0 -> 52.7 ms for 100k pairs on 256^3).
                const bool wlive = __any_sync(0xffffffffu, live);
                const float2 rsc = f2(vrow != kZeroExp ? pow2i(vrow - SLB) : 0.0f);  // 2^(row exponent - SLB)
#pragma unroll 1
                for (int c = 0; c < KP / 8; c++) {
                    if (8 * c >= L || !wlive) break;  // uniform: S columns alpha >= L are not read
                    uint32_t ra[8], rb[8], r3[8], r4[8], r5[8];
                    tc::tmem_ld8(tbase + 8 * c, ra);
                    tc::tmem_ld8(tbase + 16 + 8 * c, rb);
                    tc::tmem_ld8(tbase + 32 + 8 * c, r3);
                    tc::tmem_ld8(tbase + 48 + 8 * c, r4);
                    tc::tmem_ld8(tbase + 64 + 8 * c, r5);
                    tc::tmem_wait_ld32(ra, rb, r3, r4);
                    tc::tmem_wait_ld8(r5);  // (one wait covers all loads; the second only orders r5's use)
#pragma unroll
                    for (int i = 0; i < 4; i++) {  // two alpha per instruction
                        if (8 * c + 2 * i >= L) break;  // (L <= kNPow)
                        auto two = [&](const uint32_t *r) {
                            return make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
                        };
                        const ff2 d2 = two_sum2(two(ra), two(rb));
                        ff2 t = two_sum2(d2.hi, f2_mul(two(r3), f2(0.0009765625f)));
                        t.lo = f2_add(t.lo, f2_fma(two(r4), f2(9.5367431640625e-07f),
                                                   f2_fma(two(r5), f2(9.313225746154785e-10f), d2.lo)));
                        t = fast_two_sum2(t.hi, t.lo);
                        const float2 g = *reinterpret_cast<const float2 *>(&sm.gsc[8 * c + 2 * i]);
                        const float2 sp = f2_mul(rsc, g);
                        const float2 scl = make_float2(fminf(sp.x, 1.7014118e38f), fminf(sp.y, 1.7014118e38f));
                        float2 sh2 = f2_mul(t.hi, scl), sl2 = f2_mul(t.lo, scl);
                        if (!live) sh2 = sl2 = f2(0.0f);
                        const int a = 8 * c + 2 * i;
                        sm.st.Sh[a][m] = sh2.x;
                        sm.st.Sl[a][m] = sl2.x;
                        if (a + 1 < kNPow) {
                            sm.st.Sh[a + 1][m] = sh2.y;
                            sm.st.Sl[a + 1][m] = sl2.y;
                        }
                    }
                }
                tc::fence_before_sync();
                __syncwarp();
                // stage 2 transposed: T[z][(b,a)] = sum_y S[(z,y)][a] Y[b][y], by the warp whose
                // rows have this z (a warp barrier after the readout suffices); two partial
                // sums, over even and odd y, as one packed sum
                const int lzw = 5 - sh.ly;  // log2 of the z values per warp
                const int zbase = (warp * 32) >> sh.ly;
                // T: pass p of a warp's (q, z) in its 32 columns of S's row lp - p, which its later
                // (b, a) don't read: the pairs with b <= p, the only ones with a = lp - p, are
                // among the first 16 (p + 1)
                int row = lp;
                const int nt = npair << lzw;
                for (int t0 = 0; t0 < nt; t0 += 32, row--) {
                    if (!wlive) {
                        sm.st.Sh[row][m] = sm.st.Sl[row][m] = 0.0f;
                        continue;
                    }
                    const int t = min(t0 + (tid & 31), nt - 1);  // (all lanes come to the warp barrier)
                    const int zz = zbase + (t & ((1 << lzw) - 1));
                    const int q = t >> lzw;  // index of (b, a), rows of constant b
                    const uint32_t de = __ldg(&d_decode.e[d_decode_at(lp) + q]);  // (0, b, a)
                    const int b = (de >> 4) & 15, a = (de >> 8) & 15;
                    const float4 *ph = reinterpret_cast<const float4 *>(&sm.st.Sh[a][zz * TY]);
                    const float4 *pl = reinterpret_cast<const float4 *>(&sm.st.Sl[a][zz * TY]);
                    const float4 *yh = reinterpret_cast<const float4 *>(sm.Yh[b]);
                    const float4 *ynh = reinterpret_cast<const float4 *>(sm.Ynh[b]);
                    const float4 *ynl = reinterpret_cast<const float4 *>(sm.Ynl[b]);
                    ff2 s = {f2(0.0f), f2(0.0f)};
#pragma unroll kGeneral ? 1 : 4
                    for (int y4 = 0; y4 < TY / 4; y4++) acc_four(s, ph[y4], pl[y4], yh[y4], ynh[y4], ynl[y4]);
                    const ff r = ff_add(ff{s.hi.x, s.lo.x}, ff{s.hi.y, s.lo.y});
                    __syncwarp();  // the pass's reads of S come first
                    sm.st.Sh[row][m] = r.hi;
                    sm.st.Sl[row][m] = r.lo;
                }
                if constexpr (!kGeneral) cp_async_wait_all();  // A rows restored for the next item, masked after this
                __syncthreads();
                if (cm.abort) break;  // uniform: set before this barrier or after the next one
                lp_done = lp;
                mom_done = A.mom + moff;
            }
        }
        if (cm.abort) break;
        // the last item's (the next tile starts with a barrier)
        if (warp >= 1 && lp_done >= 0)
            add_moments(sm, mom_done, lp_done, (int)((it1 - 1 - it0) & 1), sh, warp == 1 ? tid + 32 : tid - 64);
    }
    tc_teardown(cm, kCols, phase);
}

// the float-float coefficients of every orthorhombic pair into its blob; one warp per pair
__global__ void k_coef_to_blob(const double *__restrict__ c, uint4 *blob, const int64_t *__restrict__ off16,
                               int64_t ntask) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t k = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); k < ntask; k += nw) {
        const TPair *p = reinterpret_cast<const TPair *>(blob + off16[k]);
        const int64_t src = p->coef_off;
        const int lp = p->lp;
        const int nc = ncoef(lp);
        float2 *dst = reinterpret_cast<float2 *>(blob + off16[k] + kHdr16);
        // general cell: lattice-index powers di^a dj^b dk^g -> powers of t_d = d_d |v_d|
        double hinv[3] = {1.0, 1.0, 1.0};
        if (p->general)
            for (int d = 0; d < 3; d++) hinv[d] = 1.0 / ((double)p->h[d].hi + (double)p->h[d].lo);
        for (int t = lane; t < nc; t += 32) {
            double d = c[src + t];
            if (p->general) {
                int g = 0, b = 0, r = t;
                for (g = 0; g <= lp; g++) {
                    const int cnt = ((lp - g + 1) * (lp - g + 2)) / 2;
                    if (r < cnt) break;
                    r -= cnt;
                }
                for (b = 0; b <= lp - g; b++) {
                    if (r <= lp - g - b) break;
                    r -= lp - g - b + 1;
                }
                for (int e = 0; e < g; e++) d *= hinv[2];
                for (int e = 0; e < b; e++) d *= hinv[1];
                for (int e = 0; e < r; e++) d *= hinv[0];
            }
            const float h = __double2float_rn(d);
            dst[t] = make_float2(h, __double2float_rn(d - (double)h));
        }
    }
}

// General-cell pairs [k0, k1) of an integrate call: the summed moments, in powers of
// t_d = d_d |v_d|, to powers of the lattice indices d_d; one warp per pair.  (As FP64
// products of every item's sums, up to 3 lp of them in line at 17 cycles a warp, they
// were a fifth of the integrate kernel.)
__global__ void k_scale_moments(double *mom, const uint4 *__restrict__ blob, const int64_t *__restrict__ off16,
                                int64_t k0, int64_t k1) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t k = k0 + blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); k < k1; k += nw) {
        const TPair *p = reinterpret_cast<const TPair *>(blob + off16[k]);
        double *w = mom + p->coef_off;
        const int lp = p->lp, nc = ncoef(lp);
        for (int t = lane; t < nc; t += 32) {
            const uint32_t de = __ldg(&d_decode.e[d_decode_at(lp) + t]);  // (g, b, a) of packed index t
            double v = w[t];
            for (int e = de >> 8 & 15; e > 0; e--) v *= p->hx;
            for (int e = de >> 4 & 15; e > 0; e--) v *= p->hy;
            for (int e = de & 15; e > 0; e--) v *= p->hz;
            w[t] = v;
        }
    }
}

// the image state of every item from its offsets (left in im.o by the binning),
// once per task set; one block per work unit
__global__ void k_item_images(const TileDesc *__restrict__ tiles, const int64_t *__restrict__ start,
                              const uint64_t *__restrict__ items, const uint4 *__restrict__ blob,
                              const LevelDev *__restrict__ levels, ItemImg *out, int ntiles) {
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const TileDesc td = tiles[tile];
        const int ext_x = min(TX, levels[td.level].ngrid[0] - td.t[0] * TX);
        for (int64_t it = start[2 * tile] + threadIdx.x; it < start[2 * tile + 1]; it += blockDim.x) {
            const TPair &p = *reinterpret_cast<const TPair *>(blob + (items[it] >> 16));
            ItemImg r = out[it];
            set_image_x(p, r.im, r.im.o[0], ext_x);
            out[it] = r;
        }
    }
}

// tiled calls on a task set with pairs that the binning left out
__global__ void k_report(int *status, int bits) { atomicOr(status, bits); }

// ---------------------------------------------------------------------------
// Binning on the device: the (tile, pair) items of every binned pair.
struct BinLevel {
    double G[3][3];     // metric of the lattice steps, G_ab = v_a . v_b (general cells)
    double plane[3];    // |r|^2 >= plane[a] d_a^2 whatever the other two (1 / (G^-1)_aa)
    int first;          // index of the level's first tile
    int nt[3];          // tiles per axis
    int lz;             // log2 of the tile z extent
};

// Minimum of d^T G d over the box lo <= d <= hi (G symmetric positive definite;
// infinite bounds allowed).  The minimiser has every coordinate either free or
// at one of its bounds; for each such pattern the stationary point of the free
// coordinates is solved and, if it lies in the box, its value kept.  Rounding
// can only accept a point just outside the box, which lowers the result: a test
// "minimum > r^2" built on it never drops a point inside the sphere.
__device__ double box_min_q(const double (&G)[3][3], const double (&lo)[3], const double (&hi)[3]) {
    if (lo[0] <= 0.0 && hi[0] >= 0.0 && lo[1] <= 0.0 && hi[1] >= 0.0 && lo[2] <= 0.0 && hi[2] >= 0.0) return 0.0;
    double best = HUGE_VAL;
    for (int pat = 1; pat < 27; pat++) {  // pattern 0 (all free) is the origin, handled above
        const int s[3] = {pat % 3, (pat / 3) % 3, pat / 9};  // 0 free, 1 at lo, 2 at hi
        double d[3] = {0.0, 0.0, 0.0};
        int fr[2], nf = 0;
        bool ok = true;
        for (int a = 0; a < 3; a++) {
            if (s[a] == 0) {
                fr[nf++] = a;
            } else {
                d[a] = s[a] == 1 ? lo[a] : hi[a];
                ok = ok && isfinite(d[a]);
            }
        }
        if (!ok) continue;
        auto rhs = [&](int a) {  // -(G_aX d_X) over the fixed coordinates
            double r = 0.0;
            for (int b = 0; b < 3; b++)
                if (s[b] != 0) r -= G[a][b] * d[b];
            return r;
        };
        if (nf == 1) {
            d[fr[0]] = rhs(fr[0]) / G[fr[0]][fr[0]];
        } else if (nf == 2) {
            const int a = fr[0], b = fr[1];
            const double ra = rhs(a), rb = rhs(b);
            const double det = G[a][a] * G[b][b] - G[a][b] * G[a][b];
            d[a] = (ra * G[b][b] - rb * G[a][b]) / det;
            d[b] = (G[a][a] * rb - G[a][b] * ra) / det;
        }
        for (int k = 0; k < nf; k++) {
            const int a = fr[k];
            const double tol = 1e-9 * (1.0 + fabs(d[a]));
            ok = ok && d[a] >= lo[a] - tol && d[a] <= hi[a] + tol;
        }
        if (!ok) continue;
        double q = 0.0;
        for (int a = 0; a < 3; a++)
            for (int b = 0; b < 3; b++) q += d[a] * G[a][b] * d[b];
        best = fmin(best, q);
    }
    return best;
}

// One axis of a pair's cube (cube offsets lb..hi around cc, as grid_base_ref_c.cc:318-351
// maps them) cut into runs of consecutive grid indices inside one tile.  The runs
// into one tile are the cube's periodic images over it, one item each.  Run r is the
// (t0 + r)-th tile counted through the wraps of a periodic axis.
struct AxisRuns {
    int lb, hi, T, N, nt, o0, t0, n;  // o0: cube offset of tile 0's origin (first wrap); n runs
    __device__ void init(const LevelDev &lv, int d, int cc, int lb_, int hi_, int T_, int nt_) {
        lb = lb_; hi = hi_; T = T_; nt = nt_; N = lv.ngrid[d];
        int w = lv.periodic[d] ? imod(cc + lb, lv.npts[d]) : imod(cc + lb + lv.lb_grid[d], lv.npts[d]);
        o0 = lb - w;
        if (!lv.periodic[d]) {  // points outside the window belong to no tile
            lb = max(lb, o0);
            hi = min(hi, o0 + N - 1);
            w = lb - o0;
        }
        t0 = w / T;
        const int we = hi - o0, k = we / N;
        n = hi < lb ? 0 : k * nt + (we - k * N) / T - t0 + 1;
    }
    // run r: its tile, its offsets g0..g1 and the cube offset o of the tile's origin
    __device__ __forceinline__ void get(int r, int &t, int &g0, int &g1, int &o) const {
        const int q = t0 + r, k = q < nt ? 0 : q / nt;
        t = q - k * nt;
        o = o0 + t * T + k * N;
        g0 = max(lb, o);
        g1 = min(hi, o + min(T, N - t * T) - 1);
    }
};
// the smallest folded offset |f| (f = g <= 0 ? -g : g - 1) of a run
__device__ __forceinline__ int run_fold(int a, int b) { return (a <= 1 && b >= 0) ? 0 : (b < 0 ? -b : a - 1); }

// Pass 0: items per tile (count).  Pass 1: item words and image offsets into the
// tile's slots (cursor).  A pair's image visits a tile only if some cube point of
// the image in the tile can be inside its sphere (with a margin): orthorhombic, the
// folded distance of the runs' nearest offsets <= radius; general cell, the least
// |r - rp|^2 over the lattice-index box of the runs (box_min_q) <= radius^2, tested
// per axis, then per item.  Explicit cube lists are not culled.  A pair of which some tile
// sees more than kMaxImages images along an axis gets no items: *over is set.
// kGen: the general-cell pairs [k0, k1) (the culling's box minimum needs registers
// and stack that would slow the orthorhombic launch, kGen = false).
// 2^lper threads share a pair, each on its own (z, y) runs: the largest cubes have
// hundreds of them, and few pairs alone would leave the chip idle (8000 general-cell
// pairs, one thread each, took 0.4 s to bin).
template <bool kGen>
__global__ void k_bin_pairs(const PairGeom *__restrict__ geoms, int64_t k0, int64_t k1, int lper,
                            const LevelDev *__restrict__ levels, const BinLevel *__restrict__ bl,
                            const int64_t *__restrict__ off16, const int *__restrict__ len16, int pass, int *count,
                            int *over, unsigned long long *cursor, uint64_t *items, ItemImg *iimg) {
    const int mask = (1 << lper) - 1;
    for (int64_t k = k0 + ((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> lper); k < k1;
         k += ((int64_t)gridDim.x * blockDim.x) >> lper) {
        const PairGeom &g = geoms[k];
        const LevelDev &lv = levels[g.level];
        const BinLevel B = bl[g.level];
        const TileShape sh(B.lz);
        int lb[3], hi[3];
        for (int d = 0; d < 3; d++) {  // general cell: the index box as a box-relative cube [0, hi - cc]
            lb[d] = g.ortho ? g.lb[d] : 0;
            hi[d] = g.ortho ? g.hi[d] : g.hi[d] - g.cc[d];
        }
        AxisRuns ax, ay, az;
        ax.init(lv, 0, g.cc[0], lb[0], hi[0], TX, B.nt[0]);
        ay.init(lv, 1, g.cc[1], lb[1], hi[1], sh.TY, B.nt[1]);
        az.init(lv, 2, g.cc[2], lb[2], hi[2], sh.TZ, B.nt[2]);
        if (ax.n > kMaxImages * B.nt[0] || ay.n > kMaxImages * B.nt[1] || az.n > kMaxImages * B.nt[2]) {
            *over = 1;
            continue;
        }
        int tx, ty, tz, x0, x1, y0, y1, z0, z1, ox, oy, oz;
        const double r2 = g.radius * g.radius * (1.0 + 1e-9) + 1e-12;
        const double hx = lv.dh[0][0], hy = lv.dh[1][1], hz = lv.dh[2][2];
        const bool table = g.table_off >= 0;
        const uint64_t word = ((uint64_t)off16[k] << 16) | (uint64_t)len16[k];
        auto emit = [&]() {
            const int tile = B.first + (tz * B.nt[1] + ty) * B.nt[0] + tx;
            if (pass == 0) {
                atomicAdd(count + tile, 1);
                return;
            }
            const unsigned long long at = atomicAdd(cursor + tile, 1ull);
            items[at] = word;
            iimg[at].im.o[0] = ox;
            iimg[at].im.o[1] = oy;
            iimg[at].im.o[2] = oz;
        };
        if constexpr (kGen) {
            // lattice-index offsets from the product centre: d_a = cc_a + gg - gp_a
            const double c[3] = {g.off[0] - g.cc[0], g.off[1] - g.cc[1], g.off[2] - g.cc[2]};
            const double rt = tiled_radius(g), rg = rt * rt * (1.0 + 1e-6) + 1e-12;
            double lo[3], up[3];
            auto set = [&](int a, int g0, int g1) {  // false: the run's slab lies outside the sphere
                lo[a] = g0 - c[a];
                up[a] = g1 - c[a];
                const double d = lo[a] > 0.0 ? lo[a] : (up[a] < 0.0 ? up[a] : 0.0);
                return B.plane[a] * d * d <= rg;
            };
            auto meets = [&]() {  // the box's least |r|^2 <= rg: its point nearest in indices is an upper bound
                double p[3], q = 0.0;
                for (int a = 0; a < 3; a++) p[a] = fmin(fmax(0.0, lo[a]), up[a]);
                for (int a = 0; a < 3; a++)
                    for (int b = 0; b < 3; b++) q += p[a] * B.G[a][b] * p[b];
                return q <= rg || box_min_q(B.G, lo, up) <= rg;
            };
            for (int zy = threadIdx.x & mask; zy < az.n * ay.n; zy += mask + 1) {
                const int rz = zy / ay.n;
                az.get(rz, tz, z0, z1, oz);
                ay.get(zy - rz * ay.n, ty, y0, y1, oy);
                if (!set(2, z0, z1) || !set(1, y0, y1)) continue;
                for (int rx = 0; rx < ax.n; rx++) {
                    ax.get(rx, tx, x0, x1, ox);
                    if (set(0, x0, x1) && meets()) emit();
                }
            }
        } else {
            for (int zy = threadIdx.x & mask; zy < az.n * ay.n; zy += mask + 1) {
                const int rz = zy / ay.n;
                az.get(rz, tz, z0, z1, oz);
                ay.get(zy - rz * ay.n, ty, y0, y1, oy);
                const double dz = run_fold(z0, z1) * hz, dy = run_fold(y0, y1) * hy;
                if (!table && dz * dz + dy * dy > r2) continue;
                for (int rx = 0; rx < ax.n; rx++) {
                    ax.get(rx, tx, x0, x1, ox);
                    const double dx = run_fold(x0, x1) * hx;
                    if (table || dz * dz + dy * dy + dx * dx <= r2) emit();
                }
            }
        }
    }
}

// both kinds of pairs of a task set (orthorhombic first in the sorted order)
static cudaError_t bin_pairs(const TaskSet &ts, const MixedState &M, int pass, int *count, int *over,
                             unsigned long long *cursor, uint64_t *items, ItemImg *iimg) {
    const Plan &P = *ts.plan;
    auto blocks = [](int64_t threads) {
        return (unsigned)std::max<int64_t>(1, std::min<int64_t>((threads + 127) / 128, 8192));
    };
    // about 2^18 threads (the chip's 152 SMs hold 1.2 waves of them) or one per pair
    auto share = [](int64_t n) {
        int l = 0;
        while (l < 5 && (n << l) < (1 << 18)) l++;
        return l;
    };
    if (M.northo > 0) {
        const int l = share(M.northo);
        k_bin_pairs<false><<<blocks((int64_t)M.northo << l), 128>>>(ts.d_geom, 0, M.northo, l, P.d_levels, M.d_bl,
                                                                  M.d_blob_off, M.d_blob_len, pass, count, over, cursor,
                                                                  items, iimg);
    }
    if (M.nbin > M.northo) {
        const int l = share(M.nbin - M.northo);
        k_bin_pairs<true><<<blocks((M.nbin - M.northo) << l), 128>>>(ts.d_geom, M.northo, M.nbin, l, P.d_levels,
                                                                   M.d_bl, M.d_blob_off, M.d_blob_len, pass, count, over,
                                                                   cursor, items, iimg);
    }
    return cudaGetLastError();
}

// The record (TPair) of every binned pair from its geometry, into its blob.
__global__ void k_make_records(const PairGeom *__restrict__ geoms, int64_t nbin, const LevelDev *__restrict__ levels,
                               const int64_t *__restrict__ off16, uint4 *blob) {
    auto split = [](double d) {
        const float h = __double2float_rn(d);
        return ff{h, __double2float_rn(d - (double)h)};
    };
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nbin; k += (int64_t)gridDim.x * blockDim.x) {
        const PairGeom &g = geoms[k];
        const LevelDev &lv = levels[g.level];
        TPair p;
        memset(&p, 0, sizeof p);
        const double radius = g.ortho ? g.radius : tiled_radius(g);
        p.r2 = rmul(radius, radius);
        p.r2f = __double2float_rn(p.r2);
        p.zetp = split(g.zetp);
        p.lp = g.lp;
        p.L = g.lp + 1;
        p.coef_off = g.coef_off;
        if (!g.ortho) {
            // general cell: t_d = (index_d - gp_d) |v_d|, the box as a cube [0, hi - cc] at cc
            p.general = 1;
            double len[3];
            for (int d = 0; d < 3; d++)
                len[d] = rsqrt_rn(radd(radd(rmul(lv.dh[d][0], lv.dh[d][0]), rmul(lv.dh[d][1], lv.dh[d][1])),
                                       rmul(lv.dh[d][2], lv.dh[d][2])));
            p.hx = rdiv(1.0, len[0]);
            p.hy = rdiv(1.0, len[1]);
            p.hz = rdiv(1.0, len[2]);
            p.radius = radius;
            for (int d = 0; d < 3; d++) {
                p.h[d] = split(len[d]);
                p.off[d] = split(rmul(rsub(g.off[d], (double)g.cc[d]), len[d]));
                p.lb[d] = 0;
                p.hi[d] = g.hi[d] - g.cc[d];
                p.cc[d] = g.cc[d];
                p.gp[d] = g.off[d];
                p.gpf[d] = (float)(g.off[d] - (double)p.cc[d]);
            }
            p.table_off = -1;
        } else {
            p.hx = lv.dh[0][0];
            p.hy = lv.dh[1][1];
            p.hz = lv.dh[2][2];
            p.hxf = __double2float_rn(p.hx);
            p.hyf = __double2float_rn(p.hy);
            p.hzf = __double2float_rn(p.hz);
            p.hyinvf = __double2float_rn(rdiv(1.0, p.hy));
            p.hxinvf = __double2float_rn(rdiv(1.0, p.hx));
            for (int d = 0; d < 3; d++) {
                p.off[d] = split(g.off[d]);
                p.h[d] = split(lv.dh[d][d]);
                p.lb[d] = g.lb[d];
                p.hi[d] = g.hi[d];
                p.cc[d] = g.cc[d];
            }
            p.kgmin = g.kgmin;
            p.table_off = g.table_off;
        }
        const uint4 *src = reinterpret_cast<const uint4 *>(&p);
        uint4 *dst = blob + off16[k];
        for (int c = 0; c < (int)(sizeof(TPair) / 16); c++) dst[c] = src[c];
        if (sizeof(TPair) % 16) {  // the record's last partial chunk
            uint4 last = make_uint4(0, 0, 0, 0);
            memcpy(&last, reinterpret_cast<const char *>(&p) + (sizeof(TPair) / 16) * 16, sizeof(TPair) % 16);
            dst[sizeof(TPair) / 16] = last;
        }
    }
}

int mixed_build(TaskSet &ts, std::string &err) {
    MixedState *M = new MixedState();
    ts.mixed = M;
    const Plan &P = *ts.plan;
    int64_t northo = 0;
    while (northo < ts.ntasks && ts.h_geom[northo].ortho) northo++;
    M->northo = (int)northo;
    // General-cell levels go on the tiled kernels when the cosine matrix C of the
    // lattice steps satisfies C >= 0.4 I: then sum t_d^2 <= 2.5 r^2, so inside the
    // cube the cross factor exp(-2 zetp sum c_de t_d t_e) = exp(zetp (sum t_d^2 -
    // r^2)) of the Gaussian stays within exp(69) (tiled_radius).  Otherwise they stay on the float-float
    // general kernel.
    std::vector<GenLevel> glv(P.nlevels);
    bool gen_ok = true;
    for (int l = 0; l < P.nlevels; l++) {
        const LevelDev &lv = P.lv[l];
        if (lv.ortho) continue;
        double G[3][3], h[3];
        for (int a = 0; a < 3; a++)
            for (int b = 0; b < 3; b++)
                G[a][b] = lv.dh[a][0] * lv.dh[b][0] + lv.dh[a][1] * lv.dh[b][1] + lv.dh[a][2] * lv.dh[b][2];
        for (int a = 0; a < 3; a++) h[a] = std::sqrt(G[a][a]);
        double C[3][3];
        for (int a = 0; a < 3; a++)
            for (int b = 0; b < 3; b++) C[a][b] = G[a][b] / (h[a] * h[b]) - (a == b ? 0.4 : 0.0);
        const double m1 = C[0][0], m2 = C[0][0] * C[1][1] - C[0][1] * C[1][0];
        const double m3 = C[0][0] * (C[1][1] * C[2][2] - C[1][2] * C[2][1]) -
                          C[0][1] * (C[1][0] * C[2][2] - C[1][2] * C[2][0]) +
                          C[0][2] * (C[1][0] * C[2][1] - C[1][1] * C[2][0]);
        if (!(m1 > 0.0 && m2 > 0.0 && m3 > 0.0)) gen_ok = false;
        GenLevel &q = glv[l];
        general_row_constants(lv.dh, q.row, q.rowff);
        auto sp = [](double d) {
            const float hi = (float)d;
            return ff{hi, (float)(d - (double)hi)};
        };
        q.c01 = sp(G[0][1] / (h[0] * h[1]));
        q.c02 = sp(G[0][2] / (h[0] * h[2]));
        q.c12 = sp(G[1][2] / (h[1] * h[2]));
    }
    const int64_t ngen = ts.ntasks - northo;
    // ... when every general level has a tile shape (not kUntiled) ...
    for (int l = 0; l < P.nlevels; l++)
        if (!P.lv[l].ortho && ts.tile_lz[l] == kUntiled) gen_ok = false;
    // ... and when no general box has more than kMaxImages periodic images over one tile
    // axis: count <= (extent + T - 1) / N + 1
    for (int64_t k = northo; k < ts.ntasks && gen_ok; k++) {
        const PairGeom &g = ts.h_geom[k];
        const LevelDev &lv = P.lv[g.level];
        const TileShape sh(ts.tile_lz[g.level]);
        const int T[3] = {TX, sh.TY, sh.TZ};
        for (int d = 0; d < 3; d++)
            if (lv.periodic[d] && (g.hi[d] - g.cc[d] + 1) + T[d] - 1 > (kMaxImages - 1) * lv.npts[d]) gen_ok = false;
    }
    M->gen_tiled = gen_ok && ngen > 0;
    const int64_t nbin = northo + (M->gen_tiled ? ngen : 0);
    M->nbin = nbin;
    std::vector<char> binned_level(P.nlevels, 0);
    for (int64_t k = 0; k < nbin; k++) binned_level[ts.h_geom[k].level] = 1;
    // tiles of every level with binned pairs: orthorhombic levels first
    std::vector<int> lvl_first(P.nlevels, -1);
    std::vector<TileDesc> tiles;
    int ntx[GPW_MAX_LEVELS], nty[GPW_MAX_LEVELS], ntz[GPW_MAX_LEVELS];
    for (int pass = 0; pass < 2; pass++)
    for (int l = 0; l < P.nlevels; l++) {
        if ((pass == 0) != (P.lv[l].ortho != 0)) continue;
        if (!P.lv[l].ortho && !binned_level[l]) continue;
        ntx[l] = (P.lv[l].ngrid[0] + TX - 1) / TX;
        const TileShape sh(ts.tile_lz[l]);
        nty[l] = (P.lv[l].ngrid[1] + sh.TY - 1) / sh.TY;
        ntz[l] = (P.lv[l].ngrid[2] + sh.TZ - 1) / sh.TZ;
        lvl_first[l] = (int)tiles.size();
        for (int a = 0; a < ntz[l]; a++)
            for (int b = 0; b < nty[l]; b++)
                for (int c = 0; c < ntx[l]; c++) tiles.push_back(TileDesc{l, {c, b, a}, ts.tile_lz[l], 0});
    }
    M->h_tiles = tiles;
    std::vector<BinLevel> blv(P.nlevels);
    for (int l = 0; l < P.nlevels; l++) {
        blv[l].first = lvl_first[l];
        blv[l].nt[0] = lvl_first[l] >= 0 ? ntx[l] : 0;
        blv[l].nt[1] = lvl_first[l] >= 0 ? nty[l] : 0;
        blv[l].nt[2] = lvl_first[l] >= 0 ? ntz[l] : 0;
        blv[l].lz = ts.tile_lz[l] >= 0 ? ts.tile_lz[l] : kDefaultTileLz;
        const LevelDev &lv = P.lv[l];
        for (int a = 0; a < 3; a++)
            for (int b = 0; b < 3; b++)
                blv[l].G[a][b] = lv.dh[a][0] * lv.dh[b][0] + lv.dh[a][1] * lv.dh[b][1] + lv.dh[a][2] * lv.dh[b][2];
        const double(&G)[3][3] = blv[l].G;
        const double det = G[0][0] * (G[1][1] * G[2][2] - G[1][2] * G[1][2]) -
                           G[0][1] * (G[0][1] * G[2][2] - G[1][2] * G[0][2]) +
                           G[0][2] * (G[0][1] * G[1][2] - G[1][1] * G[0][2]);
        for (int a = 0; a < 3; a++) {
            const int b = (a + 1) % 3, c = (a + 2) % 3;
            blv[l].plane[a] = det / (G[b][b] * G[c][c] - G[b][c] * G[b][c]);
        }
    }
    const int ntiles = (int)tiles.size();
    // blob layout: per task the record, then its coefficients
    std::vector<int64_t> off16((size_t)std::max<int64_t>(nbin, 1), 0);
    std::vector<int> len16((size_t)std::max<int64_t>(nbin, 1), 0);
    int64_t nchunks = 0;
    for (int64_t k = 0; k < nbin; k++) {
        off16[k] = nchunks;
        len16[k] = kHdr16 + (ncoef(ts.h_geom[k].lp) * (int)sizeof(float2) + 15) / 16;
        nchunks += len16[k];
    }
    cudaError_t e = cudaSuccess;
    auto alloc = [&](void **p, size_t bytes) {
        if (e == cudaSuccess) e = cudaMalloc(p, std::max<size_t>(bytes, 16));
    };
    alloc((void **)&M->d_blob, sizeof(uint4) * (size_t)std::max<int64_t>(nchunks, 1));
    alloc((void **)&M->d_blob_off, sizeof(int64_t) * off16.size());
    alloc((void **)&M->d_blob_len, sizeof(int) * len16.size());
    alloc((void **)&M->d_bl, sizeof(BinLevel) * blv.size());
    alloc((void **)&M->d_count, sizeof(int) * ((size_t)ntiles + 1));
    alloc((void **)&M->d_queue, sizeof(int) * 4);
    alloc((void **)&M->d_glv, sizeof(GenLevel) * glv.size());
    if (e == cudaSuccess) e = cudaMemset(M->d_blob, 0, sizeof(uint4) * (size_t)std::max<int64_t>(nchunks, 1));
    if (e == cudaSuccess)
        e = cudaMemcpy(M->d_blob_off, off16.data(), sizeof(int64_t) * off16.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess)
        e = cudaMemcpy(M->d_blob_len, len16.data(), sizeof(int) * len16.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(M->d_bl, blv.data(), sizeof(BinLevel) * blv.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess)
        e = cudaMemcpy(M->d_glv, glv.data(), sizeof(GenLevel) * glv.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(M->d_queue, 0, sizeof(int) * 4);
    if (e != cudaSuccess) {
        err = std::string("mixed_build: ") + cudaGetErrorString(e);
        return GPW_ERR_CUDA;
    }
    int sms = 0, per_sm = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, P.device);
    const void *kc[2] = {(const void *)k_collocate_tiled<false>, (const void *)k_collocate_tiled<true>};
    const void *ki[2] = {(const void *)k_integrate_tiled<false>, (const void *)k_integrate_tiled<true>};
    for (int v = 0; v < 2 && e == cudaSuccess; v++) {
        e = cudaFuncSetAttribute(kc[v], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmemColl));
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(ki[v], cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(SmemInt));
    }
    if (e != cudaSuccess) {
        err = std::string("mixed_build: ") + cudaGetErrorString(e);
        return GPW_ERR_CUDA;
    }
    // resident CTAs per SM from the kernels' own resources; TMEM (128 of 512
    // columns per CTA) caps it at 4
    auto resident = [&](const void *fn, size_t dyn) {
        cudaFuncAttributes fa;
        if (cudaFuncGetAttributes(&fa, fn) != cudaSuccess) return 1;
        int smem_sm = 0, regs_sm = 0;
        cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, P.device);
        cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, P.device);
        const int by_regs = regs_sm / std::max(1, ((fa.numRegs * 32 + 255) / 256) * 256 * (NTHR / 32));
        const int by_smem = (int)(smem_sm / (dyn + fa.sharedSizeBytes + 1024));
        return std::max(1, std::min({by_regs, by_smem, 4}));
    };
    per_sm = std::min(resident(kc[0], sizeof(SmemColl)), resident(kc[1], sizeof(SmemColl)));
    const int per_sm_i = resident(ki[0], sizeof(SmemInt));
    M->per_sm = per_sm;
    M->per_sm_i = per_sm_i;
    M->per_sm_ig = resident(ki[1], sizeof(SmemInt));
    M->sms = sms;
    // one V slot per resident integrate CTA
    const size_t vbytes = nbin > 0 ? sizeof(uint4) * kVSlot16 * (size_t)sms * std::max(per_sm_i, M->per_sm_ig) : 0;
    if (!ts.d_scratch) {
        ts.scratch_bytes = std::max(vbytes, sizeof(double) * (size_t)ts.fp64_slots * ncoef(ts.max_lp));
        if (ts.scratch_bytes > 0) e = cudaMalloc(&ts.d_scratch, ts.scratch_bytes);
    }
    M->d_vslot = static_cast<uint4 *>(ts.d_scratch);
    if (e == cudaSuccess && vbytes > ts.scratch_bytes) {
        e = cudaMalloc(&M->own_vslot, vbytes);
        M->d_vslot = M->own_vslot;
    }
    if (e != cudaSuccess) {
        err = std::string("mixed_build: ") + cudaGetErrorString(e);
        return GPW_ERR_CUDA;
    }
    return mixed_rebin(ts, err);
}

// Records, items, work units and item images from the task set's current device
// geometry (ts.d_geom): at creation and after a geometry update.  The tile
// grid, the blob layout and the choice of kernels stay as mixed_build made them.
int mixed_rebin(TaskSet &ts, std::string &err) {
    MixedState *M = ts.mixed;
    const Plan &P = *ts.plan;
    const int64_t nbin = M->nbin;
    const int ntiles = (int)M->h_tiles.size();
    cudaError_t e = cudaSuccess;
    auto fail = [&](cudaError_t ce) {
        err = std::string("mixed_rebin: ") + cudaGetErrorString(ce);
        return GPW_ERR_CUDA;
    };
    const unsigned nblk = (unsigned)std::max<int64_t>(1, std::min<int64_t>((nbin + 127) / 128, 8192));
    if (nbin > 0) {
        k_make_records<<<nblk, 128>>>(ts.d_geom, nbin, P.d_levels, M->d_blob_off, M->d_blob);
        if ((e = cudaGetLastError()) != cudaSuccess) return fail(e);
    }
    if ((e = cudaMemset(M->d_count, 0, sizeof(int) * ((size_t)ntiles + 1))) != cudaSuccess) return fail(e);
    int *over = M->d_count + ntiles;
    if (nbin > 0 && (e = bin_pairs(ts, *M, 0, M->d_count, over, nullptr, nullptr, nullptr)) != cudaSuccess) return fail(e);
    std::vector<int> count((size_t)ntiles + 1, 0);
    if ((e = cudaMemcpy(count.data(), M->d_count, sizeof(int) * count.size(), cudaMemcpyDeviceToHost)) != cudaSuccess)
        return fail(e);
    M->over = count[(size_t)ntiles] != 0;
    // items grouped by tile
    std::vector<int64_t> start(ntiles + 1, 0);
    for (int i = 0; i < ntiles; i++) start[i + 1] = start[i] + count[i];
    const int64_t nitems = start[ntiles];
    int nto = 0;
    while (nto < ntiles && P.lv[M->h_tiles[nto].level].ortho) nto++;
    // Work units for the persistent queue: a tile with more items than ~1/64 of
    // an even share per SM is divided into units of consecutive items (their
    // flushes add with FP64 atomics), and where that leaves fewer than about four
    // units per resident CTA, than 1/16 of it, down to 32 items (1000 pairs, 64^3, with
    // its 34,733 items in units of up to 16, 24, 32: integrate 354, 351, 323 us,
    // collocate 292, 298, 298).  Within each group
    // (orthorhombic, general) units run by decreasing work class (item counts within a
    // factor 2^(1/4) share a class), and within a class in the tiles' raster order: the
    // tiles in flight at one time then form a compact slab of the grid, so a pair's
    // record, coefficients and moments stay in L2 between the neighbouring tiles that
    // use them, while the short units still come last.
    const int64_t sms = std::max(1, M->sms);
    const int64_t target = std::max((nitems + 64 * sms - 1) / (64 * sms),
                                    std::min<int64_t>(64, std::max<int64_t>(32, nitems / (16 * sms))));
    // The queue's end: a group's last tiles, with as many items as one unit per resident
    // CTA but no more than an eighth, are divided into units of a quarter of that (at least
    // 8 items), which come last, unless as many items are in units of at most three
    // quarters of the largest by themselves.  (With and without: 100k pairs on 256^3,
    // units of 652 items, 58.2 and 59.4 ms collocate, 51.9 and 52.6 integrate; 1000 pairs on
    // 64^3 235 and 246, 261 and 263 us; three levels, whose units do differ, divided all the
    // same 3.76 and 3.74, 3.92 and 3.86 ms.)
    int64_t split[2];  // per group, the item from which on its tiles are divided finer
    for (int g = 0; g < 2; g++) {
        const int t0 = g ? nto : 0, t1 = g ? ntiles : nto;
        const int64_t n = start[t1] - start[t0], tail = std::min(n / 8, target * sms * (int64_t)M->per_sm);
        int64_t largest = 0, small = 0;
        auto unit = [&](int t) { return count[t] / ((count[t] + target - 1) / target); };
        for (int t = t0; t < t1; t++)
            if (count[t] > 0) largest = std::max<int64_t>(largest, unit(t));
        for (int t = t0; t < t1; t++)
            if (count[t] > 0 && 4 * unit(t) <= 3 * largest) small += count[t];
        split[g] = start[t1] - (small < tail ? tail : 0);
    }
    const int64_t fine = std::min(target, std::max<int64_t>(8, target / 4));
    // counting sort by (group, class, tile): a tile's units differ by at most one item
    // and take the class of the smaller
    std::vector<int> cls((size_t)std::max(ntiles, 1)), nu((size_t)std::max(ntiles, 1), 0);
    constexpr int kClasses = 4 * 64;
    std::vector<int> first(2 * kClasses + 1, 0);  // per group and class, the largest class first
    int nunits = 0, nuo = 0;
    for (int t = 0; t < ntiles; t++) {
        if (count[t] == 0) continue;
        const int64_t most = start[t] >= split[t >= nto] ? fine : target;
        nu[t] = (int)((count[t] + most - 1) / most);
        const int c = (int)std::floor(4.0 * std::log2((double)(count[t] / nu[t])));
        cls[t] = (t < nto ? 0 : kClasses) + kClasses - 1 - c;
        first[cls[t] + 1] += nu[t];
        nunits += nu[t];
        if (t < nto) nuo += nu[t];
    }
    for (int c = 0; c < 2 * kClasses; c++) first[c + 1] += first[c];
    // one image of everything the device needs: slots per tile, bounds per unit, tiles
    const size_t nslot = (size_t)std::max(ntiles, 1), nun = (size_t)std::max(nunits, 1);
    std::vector<unsigned char> image(8 * nslot + 16 * nun + sizeof(TileDesc) * nun);
    int64_t *slots = reinterpret_cast<int64_t *>(image.data()), *ubounds = slots + nslot;
    TileDesc *tiles_sorted = reinterpret_cast<TileDesc *>(ubounds + 2 * nun);
    for (int t = 0; t < ntiles; t++) {
        slots[t] = start[t];
        if (count[t] == 0) continue;
        const int64_t n = count[t];
        for (int64_t u = 0; u < nu[t]; u++) {
            const int at = first[cls[t]]++;
            tiles_sorted[at] = M->h_tiles[t];
            tiles_sorted[at].flags = nu[t] > 1 ? kUnitSplit : 0;
            ubounds[2 * at] = start[t] + n * u / nu[t];
            ubounds[2 * at + 1] = start[t] + n * (u + 1) / nu[t];
        }
    }
    // storage for the items and units (kept when large enough)
    if (nitems > M->cap_items || !M->d_items) {
        cudaFree(M->d_items);
        cudaFree(M->d_iimg);
        M->d_items = nullptr;
        M->d_iimg = nullptr;
        M->cap_items = 0;  // a failed allocation below leaves nothing to reuse
        const int64_t cap = std::max<int64_t>(nitems + nitems / 16, 1);
        if ((e = cudaMalloc(&M->d_items, sizeof(uint64_t) * cap)) != cudaSuccess) return fail(e);
        if ((e = cudaMalloc(&M->d_iimg, sizeof(ItemImg) * cap)) != cudaSuccess) return fail(e);
        M->cap_items = cap;
    }
    if ((int64_t)image.size() > M->cap_units || !M->d_units) {
        cudaFree(M->d_units);
        M->d_units = nullptr;
        M->cap_units = 0;
        const int64_t cap = (int64_t)image.size() + image.size() / 16;
        if ((e = cudaMalloc(&M->d_units, cap)) != cudaSuccess) return fail(e);
        M->cap_units = cap;
    }
    M->d_cursor = reinterpret_cast<unsigned long long *>(M->d_units);
    M->d_start = reinterpret_cast<int64_t *>(M->d_units) + nslot;
    M->d_tiles = reinterpret_cast<TileDesc *>(M->d_start + 2 * nun);
    if ((e = cudaMemcpy(M->d_units, image.data(), image.size(), cudaMemcpyHostToDevice)) != cudaSuccess) return fail(e);
    if (nbin > 0 && (e = bin_pairs(ts, *M, 1, nullptr, over, M->d_cursor, M->d_items, M->d_iimg)) != cudaSuccess) return fail(e);
    if (nitems) {
        k_item_images<<<std::max(1, std::min(nunits, 8192)), 128>>>(M->d_tiles, M->d_start, M->d_items, M->d_blob,
                                                                    P.d_levels, M->d_iimg, nunits);
        if ((e = cudaGetLastError()) != cudaSuccess) return fail(e);
    }
    if ((e = cudaDeviceSynchronize()) != cudaSuccess) return fail(e);
    M->ntiles_ortho = nuo;
    M->ntiles = nunits;
    M->nitems = nitems;
    return GPW_SUCCESS;
}

int64_t mixed_items(const TaskSet &ts) { return ts.mixed ? ts.mixed->nitems : 0; }
int64_t mixed_units(const TaskSet &ts) { return ts.mixed ? ts.mixed->ntiles : 0; }

void mixed_free(TaskSet &ts) {
    MixedState *M = ts.mixed;
    if (!M) return;
    cudaFree(M->d_units);
    cudaFree(M->d_blob);
    cudaFree(M->d_blob_off);
    cudaFree(M->d_items);
    cudaFree(M->d_iimg);
    cudaFree(M->d_queue);
    cudaFree(M->d_glv);
    cudaFree(M->own_vslot);
    cudaFree(M->d_bl);
    cudaFree(M->d_blob_len);
    cudaFree(M->d_count);
    delete M;
    ts.mixed = nullptr;
}

static MixedArgs make_args(const TaskSet &ts, const GridPtrs &g, int which, bool general) {
    const MixedState &M = *ts.mixed;
    const int t0 = general ? M.ntiles_ortho : 0;
    MixedArgs a;
    a.blob = M.d_blob;
    a.levels = ts.plan->d_levels;
    a.tiles = M.d_tiles + t0;
    a.start = M.d_start + 2 * t0;
    a.items = M.d_items;
    a.iimg = M.d_iimg;
    a.table = ts.d_table;
    a.glv = M.d_glv;
    a.mom = ts.d_mom;
    a.vslot = M.d_vslot;
    a.grids = g;
    a.queue = M.d_queue + which + (general ? 2 : 0);
    a.status = ts.d_status;
    a.ntiles = general ? M.ntiles - M.ntiles_ortho : M.ntiles_ortho;
    return a;
}

// a tiled call that lacks pairs: an error status (a plain FP64 call must not see it)
static cudaError_t report_over(const TaskSet &ts, cudaStream_t s) {
    ts.n_kernels++;
    k_report<<<1, 1, 0, s>>>(ts.d_status, kStatTooManyImages);
    return cudaGetLastError();
}

cudaError_t launch_collocate_mixed(const TaskSet &ts, const GridPtrs &g, cudaStream_t s) {
    if (!ts.mixed) return cudaErrorNotSupported;
    const MixedState &M = *ts.mixed;
    cudaError_t e = cudaSuccess;
    if (M.over && (e = report_over(ts, s)) != cudaSuccess) return e;
    if (M.nbin > 0 && M.ntiles > 0) {
        ts.n_kernels++;
        k_coef_to_blob<<<(unsigned)std::min<int64_t>((M.nbin + 7) / 8, 8192), 256, 0, s>>>(ts.d_coef, M.d_blob,
                                                                                             M.d_blob_off, M.nbin);
        const int nto = M.ntiles_ortho, ntg = M.ntiles - M.ntiles_ortho;
        if (nto > 0) {
            if ((e = cudaMemsetAsync(M.d_queue, 0, sizeof(int), s)) != cudaSuccess) return e;
            ProfScope prof(ts, s);
            k_collocate_tiled<false><<<std::min(nto, M.sms * M.per_sm), NTHR, sizeof(SmemColl), s>>>(
                make_args(ts, g, 0, false));
            if ((e = cudaGetLastError()) != cudaSuccess) return e;
        }
        if (ntg > 0) {
            if ((e = cudaMemsetAsync(M.d_queue + 2, 0, sizeof(int), s)) != cudaSuccess) return e;
            ProfScope prof(ts, s);
            k_collocate_tiled<true><<<std::min(ntg, M.sms * M.per_sm), NTHR, sizeof(SmemColl), s>>>(
                make_args(ts, g, 0, true));
            if ((e = cudaGetLastError()) != cudaSuccess) return e;
        }
    }
    return M.gen_tiled ? cudaSuccess : launch_general_ff(ts, g, false, s);
}

cudaError_t launch_integrate_mixed(const TaskSet &ts, const GridPtrs &g, cudaStream_t s) {
    if (!ts.mixed) return cudaErrorNotSupported;
    const MixedState &M = *ts.mixed;
    cudaError_t e = cudaSuccess;
    if (M.over && (e = report_over(ts, s)) != cudaSuccess) return e;
    if (M.nbin > 0) {
        if ((e = cudaMemsetAsync(ts.d_mom, 0, sizeof(double) * ts.coef_len, s)) != cudaSuccess) return e;
        const int nto = M.ntiles_ortho, ntg = M.ntiles - M.ntiles_ortho;
        if (nto > 0) {
            if ((e = cudaMemsetAsync(M.d_queue + 1, 0, sizeof(int), s)) != cudaSuccess) return e;
            ProfScope prof(ts, s);
            k_integrate_tiled<false><<<std::min(nto, M.sms * M.per_sm_i), NTHR, sizeof(SmemInt), s>>>(
                make_args(ts, g, 1, false));
            if ((e = cudaGetLastError()) != cudaSuccess) return e;
        }
        if (ntg > 0) {
            if ((e = cudaMemsetAsync(M.d_queue + 3, 0, sizeof(int), s)) != cudaSuccess) return e;
            ProfScope prof(ts, s);
            k_integrate_tiled<true><<<std::min(ntg, M.sms * M.per_sm_ig), NTHR, sizeof(SmemInt), s>>>(
                make_args(ts, g, 1, true));
            if ((e = cudaGetLastError()) != cudaSuccess) return e;
            ts.n_kernels++;
            k_scale_moments<<<(unsigned)std::min<int64_t>((M.nbin - M.northo + 7) / 8, 8192), 256, 0, s>>>(
                ts.d_mom, M.d_blob, M.d_blob_off, M.northo, M.nbin);
            if ((e = cudaGetLastError()) != cudaSuccess) return e;
        }
    }
    return M.gen_tiled ? cudaSuccess : launch_general_ff(ts, g, true, s);
}

}  // namespace gpw
