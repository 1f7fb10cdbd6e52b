// Internal declarations shared by the CUDA translation units of
// libSharedVDBSCAN.so (GB300, sm_103a).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <string>
#include <vector>

namespace vdb {

// Kernels launched by this library since it was loaded.
extern std::atomic<unsigned long long> g_launches;

// Launches go out with programmatic stream serialization: a kernel may be
// scheduled while the one before it still runs, and every kernel begins with
// pdl_sync(), which waits until that one has completed and its writes are
// visible (so the order of the work is the stream's), then lets the next one
// be scheduled.  A chain of small kernels thus does not pay each launch's
// latency in turn.  Not while a stream is captured (the thread's g_plain_launch;
// the graph's nodes depend on whole kernels).
extern thread_local bool g_plain_launch;
static __device__ __forceinline__ void pdl_sync() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <class... P, class... A>
inline void launch(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t s, A... args) {
    g_launches.fetch_add(1, std::memory_order_relaxed);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = s;
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = g_plain_launch ? 0 : 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

constexpr int kVisitBins = 300;          // src/main.cpp:107 (binDataset(&dataPoints, 300, ...))
constexpr int kMaxRows = 65;             // neighbour rows per tile: 2*rho+1 <= 65
constexpr uint32_t kAsymFlag = 0x80000000u;  // neighbour-table entry accepted in one direction only
constexpr uint32_t kIdMask = 0x7fffffffu;
// Compact tables: 16-bit entries.  A row lists its neighbours work unit by
// work unit (units of 512 to 4096 candidates of the row's tile, in
// order; the count pass's per-unit counts give each unit's share of the row);
// an entry holds the neighbour's position within its unit's candidates (12
// bits) and, in the top bit, the one-way flag.  Positions map to cell-ordered
// indices through the tile's 2*rho+1 row segments.
constexpr uint16_t kAsymFlag16 = 0x8000u;
constexpr uint16_t kPosMask16 = 0x0fffu;

// Status bits written by kernels into DeviceStatus::flags.
enum : uint32_t {
    kStatNonFinite = 1u << 0,    // NaN or inf coordinate
    kStatDegenerate = 1u << 1,   // reference binDataset would report bins out of range
    kStatAsymOverflow = 1u << 2, // asymmetric-pair list full
    kStatResolveOverflow = 1u << 3,  // too many directed component edges
    kStatRowOverflow = 1u << 4,      // fill pass found more neighbours than the count pass
    kStatUnionStall = 1u << 5,       // union-find retry limit reached
    kStatGuard = 1u << 6,            // an index guard failed (see guard_site)
    kStatBitmapTooLarge = 1u << 7,   // a tile's test bitmap exceeds 2^32 words (use the fill pass)
    kStatTooManyUnits = 1u << 8,     // 2^31 work units or more: their offsets and number are void
};

constexpr uint32_t kResolveCap = 4096;   // directed component edges per variant

struct DeviceStatus {
    uint32_t flags;
    uint32_t guard_site;           // first failed index guard: site code
    unsigned long long retested;   // FP64 re-tests
    unsigned long long candidates; // candidate pairs tested
    unsigned long long asym_count; // asymmetric pairs recorded
    unsigned long long guard_value; // first failed index guard: the index
    unsigned long long clusters;   // clusters summed over the variants written
    unsigned long long table_hash; // hash of the tables built (vdb_stats.table_hash)
    unsigned long long reuse_skips; // cell pairs not searched: different components at a
                                    // larger epsilon
    unsigned long long pairs;      // neighbour pairs counted (graph replays, labels-only calls)
    // sizes of the current epsilon, which the host reads back with the rest
    unsigned long long nwords;     // words of the test bitmap
    unsigned long long entries;    // entries of the neighbour table
    uint32_t nunits;               // work units
    uint32_t ntiles;
    uint32_t asym_n;               // one-way pairs recorded
    uint32_t starts_done[8];       // blocks done per slot of cell_starts_kernel
};

// Index guards: a data-derived index outside its array is recorded (site and
// value of the first one) and the access is skipped.
__device__ __forceinline__ void guard_fail(DeviceStatus* st, uint32_t site,
                                           unsigned long long v) {
    if (atomicOr(&st->flags, 1u << 6) & (1u << 6)) return;
    st->guard_site = site;
    st->guard_value = v;
}
#define VDB_GUARD(st, cond, site, val) ((cond) ? true : (guard_fail((st), (site), (val)), false))

// Bounding box with the reference's initial values (src/main.cpp:465-468):
// min starts at DBL_MAX, max at DBL_MIN (the smallest positive double).
struct BBox {
    double minx, maxx, miny, maxy;      // reference semantics (max >= DBL_MIN)
    double tmaxx, tmaxy;                // true maxima
    uint32_t nonfinite;
    uint32_t pad;
};

// Grid over a dataset: cells of width w (exactly representable with 12
// significant bits, so small multiples of w are exact in FP32), row-major keys
// key = cy*ncx_pad + cx.  A tile covers up to kTileQueries consecutive points of
// one group of G cells of one row.
struct GridParams {
    double x0, y0, w;
    uint32_t ncx, ncy, ncx_pad, G;
    uint64_t ncells;                    // ncx_pad*ncy
    // 0: cells are looked up in a dense cell_start array (ncells+1 entries);
    // 1: many more cells than points - a row directory of the non-empty
    //    cells (crow, ccx, clist) replaces it
    uint32_t sparse;
    // points are sorted by cell and, within a cell, along a Hilbert curve of
    // 2^sub x 2^sub subcells (neighbours in the order are near each other)
    uint32_t sub;
};

// Points [*s, *e) of the cells lo_c..hi_c of grid row ry (cell order).
// Dense grids: cell_start[key] = first point of the first non-empty cell with
// a key >= key.  Sparse grids: crow[ry]..crow[ry+1] are the non-empty cells of
// row ry (sorted by column ccx), clist[c] the first point of cell c.
static __device__ __forceinline__ uint32_t cx_lower_bound(const uint32_t* __restrict__ ccx,
                                                          uint32_t b, uint32_t e, uint32_t v) {
    while (b < e) {
        const uint32_t m = (b + e) >> 1;
        if (ccx[m] < v) b = m + 1;
        else e = m;
    }
    return b;
}
static __device__ __forceinline__ void cell_row_range(const GridParams& g,
                                                      const uint32_t* __restrict__ cell_start,
                                                      const uint32_t* __restrict__ crow,
                                                      const uint32_t* __restrict__ ccx,
                                                      const uint32_t* __restrict__ clist,
                                                      uint32_t ry, uint32_t lo_c, uint32_t hi_c,
                                                      uint32_t* s, uint32_t* e) {
    if (g.sparse) {
        const uint32_t rb = crow[ry], re = crow[ry + 1];
        const uint32_t c0 = cx_lower_bound(ccx, rb, re, lo_c);
        const uint32_t c1 = cx_lower_bound(ccx, c0, re, hi_c + 1);
        *s = clist[c0];
        *e = clist[c1];
    } else {
        const uint32_t base = ry * g.ncx_pad;
        *s = cell_start[base + lo_c];
        *e = cell_start[base + hi_c + 1];
    }
}

// Doubles as unsigned integers of the same order (-0 just below +0), and back.
// Minima and maxima are taken of these: GB300's FP64 pipe takes 16 cycles for a
// warp's comparison, the integer pipe less than 2.
static __device__ __forceinline__ unsigned long long ordered_key(double v) {
    const long long b = __double_as_longlong(v);
    return (unsigned long long)(b ^ ((b >> 63) | (long long)0x8000000000000000ull));
}
static __device__ __forceinline__ double ordered_value(unsigned long long k) {
    const long long b = (long long)k;
    return __longlong_as_double(b ^ (~(b >> 63) | (long long)0x8000000000000000ull));
}
// The largest of a warp's values (every lane, the result in all lanes).
static __device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long v) {
    const uint32_t hi = __reduce_max_sync(0xffffffffu, (uint32_t)(v >> 32));
    const uint32_t lo =
        __reduce_max_sync(0xffffffffu, (uint32_t)(v >> 32) == hi ? (uint32_t)v : 0u);
    return ((unsigned long long)hi << 32) | lo;
}

// Bounds of the exact predicate as ordered integers.  For doubles >= +0 the
// order of the values is the order of their bit patterns read as integers, so
// the predicate compares d2 and |d| with integer instructions and leaves
// GB300's narrow FP64 pipe to the subtractions and products.  A negative or
// NaN bound becomes -1, which no value passes (as with the FP64 comparison).
struct ExactBounds {
    double eps;
    long long thr, tbox, ax;  // thr, tbox and ax_in = sqrt(tbox), ordered
};

// Distance test of one epsilon.
struct EpsParams {
    double eps;
    double thr;     // largest double t with sqrt(t) <= eps
    double tbox;    // d2 <= tbox guarantees the candidate lies in the query box
    ExactBounds xb; // of eps, thr and tbox
    float wf;       // the cells' width, FP32
    float near2;    // eps^2 (1 + 2^-8), FP32
    float iw;       // 1 / the cells' width, FP32
    float lo32;     // FP32 d2 < lo32: neighbour (no FP64 re-test)
    float hi32;     // FP32 d2 > hi32: not a neighbour
    // count pass filter on the quadratic form nS = |c|^2/2 + (|q|^2 - L32)/2 - q.c
    // (= (d2 - L32)/2 up to rounding): nS < 0 => d2 < lo32 (in); nS > w32 =>
    // d2 > hi32 (out); every nS in between is re-tested in FP64
    float L32;
    float w32;
    int rho;        // rows above/below the tile row to scan
    int mixed;      // 1: FP32 filter + FP64 band re-test; 0: FP64 only
    int reach[kMaxRows];  // columns left/right of the tile's cells to scan, per row offset+rho
};

// Bounding box of one group of MBBsize consecutive visit-ordered points
// (the reference's MPBRect, src/structs.h:70-125).
struct __align__(32) MpbBox {
    double x0, x1, y0, y1;   // min x, max x, min y, max y
};

struct AsymPair {
    uint32_t a, b;     // grid indices, a < b
    uint32_t dir;      // bit0: b in N(a); bit1: a in N(b)
    uint32_t pad;
};

// ------------------------------------------------- the reference's predicate
// q in N(p)  <=>  sqrt(fl(fl(dx*dx)+fl(dy*dy))) <= eps with dx = fl(px-qx) in
// FP64 (src/DBScan.cpp:687, 699-702) and q's multiple-point box overlaps the
// query box [p-eps, p+eps]^2 (R-tree candidates, src/RTree.h:1613-1625).

// q inside the query box of p (DBScan::generateMBB, src/DBScan.cpp:722-731);
// a point inside the box makes its multiple-point box overlap it.
static __device__ __forceinline__ bool in_query_box(double qx, double qy, double px, double py,
                                                    double eps) {
    const double x0 = __dsub_rn(px, eps), x1 = __dadd_rn(px, eps);
    const double y0 = __dsub_rn(py, eps), y1 = __dadd_rn(py, eps);
    return !(x0 > qx || qx > x1 || y0 > qy || qy > y1);
}

static __device__ __forceinline__ bool box_overlap(MpbBox m, double px, double py, double eps) {
    const double x0 = __dsub_rn(px, eps), x1 = __dadd_rn(px, eps);
    const double y0 = __dsub_rn(py, eps), y1 = __dadd_rn(py, eps);
    return !(x0 > m.x1 || m.x0 > x1 || y0 > m.y1 || m.y0 > y1);
}

// Exact predicate in both directions: bit0 = q in N(p), bit1 = p in N(q).
// thr: largest double whose square root is <= eps; tbox: below it the pair is
// inside both query boxes; ax_in = sqrt(tbox): an axis along which
// |d| <= ax_in keeps each point inside the other's query box whatever the
// roundings of p +- eps (the margin behind tbox is per axis), so the box
// arithmetic is done only along the other axis.  d2 >= +0 and |d| >= +0 are
// compared as ordered integers (ExactBounds).  kp, kq: cell-ordered indices;
// gbox[k]: the multiple-point box holding cell-ordered point k (one load, no
// index chain).
static __device__ __noinline__ uint32_t exact_pair(double2 P, double2 Q, uint32_t kp,
                                                   uint32_t kq, const ExactBounds b,
                                                   const MpbBox* __restrict__ gbox) {
    const double dx = __dsub_rn(P.x, Q.x), dy = __dsub_rn(P.y, Q.y);
    const double d2 = __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy));
    const long long d2b = __double_as_longlong(d2);
    if (!(d2b <= b.thr)) return 0u;
    if (d2b <= b.tbox) return 3u;
    const long long mag = 0x7fffffffffffffffll;
    const bool inx = (__double_as_longlong(dx) & mag) <= b.ax;
    const bool iny = (__double_as_longlong(dy) & mag) <= b.ax;
    if (inx && iny) return 3u;
    const double eps = b.eps;
    uint32_t r = 0u;
    // q inside the query box of p (DBScan::generateMBB, src/DBScan.cpp:722-731)
    const bool qin = (inx || !(__dsub_rn(P.x, eps) > Q.x || Q.x > __dadd_rn(P.x, eps))) &&
                     (iny || !(__dsub_rn(P.y, eps) > Q.y || Q.y > __dadd_rn(P.y, eps)));
    if (qin || box_overlap(gbox[kq], P.x, P.y, eps)) r |= 1u;
    const bool pin = (inx || !(__dsub_rn(Q.x, eps) > P.x || P.x > __dadd_rn(Q.x, eps))) &&
                     (iny || !(__dsub_rn(Q.y, eps) > P.y || P.y > __dadd_rn(Q.y, eps)));
    if (pin || box_overlap(gbox[kp], Q.x, Q.y, eps)) r |= 2u;
    return r;
}

// Compact-table decoding, one warp per row (every lane must call both, with
// the same t): lane i < nrows holds the start of segment i of tile t's
// candidate list and the number of candidates before it.
struct TileSegs {
    uint32_t start, before;
};
static __device__ __forceinline__ TileSegs load_tile_segs(const uint32_t* __restrict__ trow_s,
                                                          const uint32_t* __restrict__ trow_e,
                                                          uint32_t t, int nrows, int lane) {
    uint32_t st = 0, len = 0;
    if (lane < nrows) {
        const unsigned long long k = (unsigned long long)t * (uint32_t)nrows + (uint32_t)lane;
        st = trow_s[k];
        len = trow_e[k] - st;
    }
    uint32_t incl = len;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += v;
    }
    return TileSegs{st, incl - len};
}
// Cell-ordered index of candidate position g (g below the tile's total).
static __device__ __forceinline__ uint32_t decode_candidate(const TileSegs& sg, int nrows,
                                                            uint32_t g) {
    uint32_t id = 0;
    for (int i = 0; i < nrows; i++) {
        const uint32_t b = __shfl_sync(0xffffffffu, sg.before, i);
        const uint32_t s0 = __shfl_sync(0xffffffffu, sg.start, i);
        if (g >= b) id = s0 + (g - b);
    }
    return id;
}

// ----------------------------------------------------------------- primitives
// All launches go to `s`.  "zeroed" memory is zero at the launch and used up
// by it.

// Exclusive scan of n uint32 values into uint64 (out has n+1 entries; out[n] =
// st->entries = total).
size_t scan_state_bytes(uint32_t n);
void scan_u32_to_u64(const uint32_t* in, unsigned long long* out, uint32_t n, void* zeroed,
                     DeviceStatus* st, cudaStream_t s);

// Stable LSD radix sort of keys and their indices on the low `bits` key bits.
// zeroed: sort_zero_bytes, its first sort_passes(bits) * kDigits words holding
// the keys' digit counts by the time of the call (the kernels that make the
// keys count them).  okeys (may be null): the sorted keys >> drop; ovals: the
// indices in key order; oinv (may be null): oinv[index] = its place.
constexpr int kDigitBits = 9;
constexpr uint32_t kDigits = 1u << kDigitBits;
constexpr int kMaxPasses = 4;
int sort_passes(int bits);
size_t sort_zero_bytes(uint32_t n, int bits);
size_t sort_scratch_bytes(uint32_t n);
void radix_sort(const uint32_t* keys, uint32_t n, int bits, int drop, void* zeroed, void* scratch,
                uint32_t* okeys, uint32_t* ovals, uint32_t* oinv, DeviceStatus* st,
                cudaStream_t s);

// ------------------------------------------------------------------ index
// (zeroed: one word)
void launch_bbox(const double* x, const double* y, uint32_t n, BBox* out, void* scratch,
                 uint32_t* zeroed, cudaStream_t s);
size_t bbox_scratch_bytes();
// keys and their digit counts (hist: sort_passes(17) * kDigits zeroed words)
constexpr int kVisitBits = 17;
void launch_visit_keys(const double* x, const double* y, uint32_t n, const BBox* bb,
                       uint32_t* keys, uint32_t* hist, DeviceStatus* st, cudaStream_t s);
void launch_mpb_boxes(const double* x, const double* y, const uint32_t* vorder, uint32_t n,
                      int mbb, MpbBox* boxes, cudaStream_t s);
// (the epsilon's parameters are left at ep_out for the kernels that follow)
void launch_grid_keys(const double* x, const double* y, uint32_t n, GridParams g, int bits,
                      uint32_t* keys, uint32_t* hist, const EpsParams& ep, EpsParams* ep_out,
                      cudaStream_t s);

// The cell order's arrays: per point the coordinates (gxy, FP32 relative to
// the own cell: glocal), visit position and multiple-point box; the non-empty
// cells (cscan[k]: cells that start before point k, clist: first points, ckey,
// ccx: keys and columns; cscan[n] = their number, clist[number] = n) and the
// tiles (tiles: first points, tiles[number] = n; ptile: tile of
// every point; *ntiles).
struct OrderArgs {
    const double* x;
    const double* y;
    const uint32_t* gorig;
    const uint32_t* pos;
    const uint32_t* gkey;
    uint32_t n;
    GridParams g;
    double2* gxy;
    float2* glocal;
    uint32_t* gpos;
    const MpbBox* mpb;
    uint32_t mbb;
    MpbBox* gbox;
    uint32_t* cscan;
    uint32_t* clist;
    uint32_t* ckey;
    uint32_t* ccx;
    uint32_t tq;                // points per tile at most
    uint32_t* tiles;
    uint32_t* ptile;
    uint32_t* ntiles;
    unsigned long long* cbest;  // cleared (n words) for cell_setup_kernel; may be null
    DeviceStatus* st;
};
size_t order_state_bytes(uint32_t n);
void launch_order(const OrderArgs& a, void* zeroed, cudaStream_t s);
// gxy, glocal, gpos, gbox alone (no grid: an epsilon without neighbours)
void launch_gather(const OrderArgs& a, cudaStream_t s);
// cell_start[key] = first point of the first non-empty cell at or after key
// (ncells + 1 entries)
void launch_cell_start(const uint32_t* ckey, const uint32_t* clist, const uint32_t* ncl,
                       uint32_t n, const GridParams& g, uint32_t* cell_start, cudaStream_t s);
// crow[r] = first non-empty cell of row >= r (ncy + 1 entries; sparse grids)
void launch_cell_rows(const uint32_t* ckey, const uint32_t* ncl, const GridParams& g,
                      uint32_t* crow, cudaStream_t s);
// ------------------------------------------------------------------ tables
struct TableArgs {
    GridParams g;
    const EpsParams* ep;        // device copy
    int mixed;                  // 1: FP32 filter kernels, 0: FP64 kernels
    const uint32_t* tiles;      // tile start indices (ntiles+1 entries, last = n)
    const uint32_t* ntiles;     // device scalar
    uint32_t tile_end;          // 0xffffffff: use *ntiles
    uint32_t* tile_counter;     // device scalar: first tile to take (set before launch)
    const uint32_t* cell_start; // ncells+1 entries (dense grids)
    const uint32_t* crow;       // sparse grids: row directory (see cell_row_range)
    const uint32_t* ccx;
    const uint32_t* clist;      // first point of each non-empty cell (ncl+1 entries)
    // sparse grids and compact tables: candidate range of row i of tile t at
    // [t*(2*rho+1) + i] (written by the tile-words pass, read by the count and
    // expand passes and, for compact tables, by every reader of the table)
    uint32_t* trow_s;
    uint32_t* trow_e;
    const uint32_t* ptile;      // compact tables: tile of every cell-ordered point
    int compact;                // nonzero: nbr holds 16-bit entries (kAsymFlag16)
    const uint32_t* gkey;
    const float2* glocal;
    const double2* gxy;
    float4* wbox;               // boxes of runs of points (launch_unit_list), (n+3)/4; may be null
    const uint32_t* gpos;
    const MpbBox* gbox;         // multiple-point box of each cell-ordered point
    uint32_t n;
    uint32_t* deg;              // count pass output
    const unsigned long long* off;  // fill pass: row offsets (n+1)
    unsigned long long off_base;    // fill pass: first entry held by nbr
    uint32_t* nbr;                  // fill pass output (uint16_t entries when compact)
    AsymPair* asym;
    uint32_t* asym_n;
    uint32_t asym_cap;
    DeviceStatus* st;
    uint32_t* bitmap;               // count pass: per-tile test bitmaps (nullptr: none)
    const unsigned long long* tile_boff;  // first bitmap word of each tile
    // work units of the count and table passes: (tile, chunk of unit_words
    // bitmap words); tile t has the units tile_uoff[t]..tile_uoff[t+1], which
    // warps take, and ulist holds their tile.  Small tiles have none: a thread
    // per point takes them, and their rows are one piece.
    uint32_t unit_words;            // bitmap words per unit (default_unit_words)
    const uint32_t* ulist;
    const uint32_t* tile_uoff;
    const uint32_t* nunits;         // device scalar
    uint32_t* parts;                // per unit and query slot: neighbours in that chunk
    uint2* wflags;                  // per unit and block of 32 words: words wholly inside eps of
                                    // the tile, wholly outside (16-bit tables; else null)
    unsigned long long* pair_sum;   // count pass: adds the neighbours counted (nullptr: not)
    // one row chunk of the table: the fill pass takes tiles from tile_lo on,
    // the expand pass units [unit_lo, unit_hi), and the small tiles
    // and the asymmetric flags touch rows [row_lo, row_hi) only
    uint32_t tile_lo;
    uint32_t unit_lo, unit_hi;
    uint32_t row_lo, row_hi;
};
// Work units hold up to 4096 candidates of a tile (kUnitWords bitmap words;
// compact entries are positions within a unit, 12 bits), down to 512
// (kUnitWordsTiny) for tables of few units (default_unit_words).
constexpr uint32_t kUnitWords = 128;
constexpr uint32_t kUnitWordsSmall = 32;
constexpr uint32_t kUnitWordsTiny = 16;
// Entries of wflags per unit.
static __host__ __device__ __forceinline__ uint32_t flag_blocks(uint32_t unit_words) {
    return (unit_words + 31u) / 32u;
}
constexpr uint32_t kUnitQ = 64;        // query slots per unit (tiles hold <= 64 queries)

// Walks row k of a compact table (nb16, the row's entries [row0, row1)) unit
// by unit, 32 entries at a time: fn(neighbour cell-ordered index, one-way
// flag, valid) on every lane (the decoding shuffles need the whole warp; lanes
// past the end get valid = false).  parts[u * kUnitQ + slot]: the row's
// entries in unit u (not looked at where the tile has one unit, or none, as small
// tiles: the row is one piece); unit_words: the table's unit size in bitmap words.
template <class Fn>
static __device__ __forceinline__ void walk_compact_row(
    const uint16_t* __restrict__ nb16, unsigned long long row0, unsigned long long row1, uint32_t k,
    const uint32_t* __restrict__ ptile, const uint32_t* __restrict__ tiles,
    const uint32_t* __restrict__ tile_uoff, const uint32_t* __restrict__ parts,
    const uint32_t* __restrict__ trow_s, const uint32_t* __restrict__ trow_e, int nrows,
    uint32_t unit_words, int lane, Fn&& fn) {
    const uint32_t t = ptile[k];
    const uint32_t slot = k - tiles[t];
    const uint32_t u0 = tile_uoff[t];
    const uint32_t u1 = max(tile_uoff[t + 1], u0 + 1u);
    const TileSegs sg = load_tile_segs(trow_s, trow_e, t, nrows, lane);
    const uint32_t len = (uint32_t)(row1 - row0);
    uint32_t j = 0;  // entries of the row before unit ub
    for (uint32_t ub = u0; ub < u1; ub += 32) {
        const uint32_t u = ub + (uint32_t)lane;
        uint32_t c = 0;
        if (u < u1 && slot < kUnitQ)
            c = u1 - u0 == 1u ? len : parts[(unsigned long long)u * kUnitQ + slot];
        uint32_t incl = c;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += v;
        }
        const uint32_t jb = j + (incl - c);
        for (uint32_t nz = __ballot_sync(0xffffffffu, c != 0u); nz; nz &= nz - 1u) {
            const int src = __ffs(nz) - 1;
            const uint32_t cu = __shfl_sync(0xffffffffu, c, src);
            const uint32_t js = __shfl_sync(0xffffffffu, jb, src);
            const uint32_t gbase = (ub + (uint32_t)src - u0) * (unit_words * 32u);
            for (uint32_t e0 = 0; e0 < cu; e0 += 32) {
                const bool valid = e0 + (uint32_t)lane < cu && js + e0 + (uint32_t)lane < len;
                const uint16_t ev = valid ? nb16[row0 + js + e0 + (uint32_t)lane] : (uint16_t)0;
                const uint32_t id = decode_candidate(sg, nrows, gbase + (ev & kPosMask16));
                fn(id, (ev & kAsymFlag16) != 0, valid);
            }
        }
        j += __shfl_sync(0xffffffffu, incl, 31);
    }
}
void launch_count(const TableArgs& a, int nblocks, cudaStream_t s);
void launch_fill(const TableArgs& a, int nblocks, cudaStream_t s);
size_t words_state_bytes(uint32_t n);
void launch_tile_words(const TableArgs& a, unsigned long long* boff, uint32_t* uoff,
                       unsigned long long* nwords, uint32_t* nunits, void* zeroed,
                       cudaStream_t s);
void launch_unit_list(const TableArgs& a, uint32_t* ulist, cudaStream_t s);
// adds the hash of rows [row_lo, row_hi) of the table to st->table_hash
// (gorig: input index of every cell-ordered point)
void launch_table_hash(const TableArgs& a, const uint32_t* gorig, int nblocks, cudaStream_t s);
void launch_expand(const TableArgs& a, int nblocks, cudaStream_t s);
void launch_asym_flags(const TableArgs& a, cudaStream_t s);

// Rows [r_lo, r_hi) of the neighbour table = tiles [t_lo, t_hi) = work units
// [u_lo, u_hi), table entries [e_lo, e_hi).  The whole
// table: t_hi = u_hi = 0xffffffff (no limits).
struct RowChunk {
    uint32_t t_lo, t_hi, u_lo, u_hi, r_lo, r_hi;
    uint64_t e_lo, e_hi;
};
constexpr uint32_t kPlanChunks = 64;
struct ChunkPlan {
    uint32_t n;       // chunks listed here
    uint32_t next;    // first tile after them
    uint32_t ntiles;
    uint32_t refused; // 1: a tile's rows exceed the cap, 2: the tile list does not end at n
    RowChunk list[kPlanChunks];
};
// The next (up to kPlanChunks) row chunks from tile t0: whole tiles, at most cap
// entries each, greedy in tile order.
void launch_plan_chunks(const uint32_t* tiles, const uint32_t* ntiles, const uint32_t* tuoff,
                        const unsigned long long* off, uint32_t n, uint64_t cap, uint32_t t0,
                        ChunkPlan* plan, cudaStream_t s);
int table_block_threads();
int table_tile_queries();
int table_blocks_per_sm(bool fill, bool mixed);
int expand_blocks_per_sm(bool compact);

// ------------------------------------------------------------------ clustering
struct ClusterArgs {
    uint32_t n;
    const uint32_t* deg;
    unsigned long long minpts;      // ~0ull: no core points
    unsigned long long minpts_prev; // ~0ull: union-find starts from scratch; else the
                                    // cores of minpts_prev are already united in parent
    const unsigned long long* off;
    unsigned long long off_base;
    uint32_t row_lo, row_hi;
    const uint32_t* nbr;        // uint16_t entries when compact
    int compact;                // compact table: entries decoded through ptile, trow_s/e,
    const uint32_t* ptile;      // the tiles' first points and work units, and the count
    const uint32_t* trow_s;     // pass's per-unit counts
    const uint32_t* trow_e;
    const uint32_t* tiles;
    const uint32_t* tile_uoff;
    const uint32_t* parts;
    uint32_t unit_words;        // the table's work-unit size in bitmap words
    const uint32_t* gpos;
    const uint32_t* gorig;
    uint32_t* parent;
    uint32_t* seed;             // per root: min visit position of its cores
    uint32_t* cstart;           // per root: root of the component that starts its cluster
    uint32_t* best;             // per point: earliest cluster start among adjacent cores
    uint32_t* bits;             // visit positions at which clusters start
    uint32_t* brank;            // starts before each word of bits
    uint32_t nw;                // start_words(n)
    const AsymPair* asym;
    const uint32_t* asym_count;
    uint32_t asym_cap;
    uint32_t* labels_out;       // n labels in input order
    DeviceStatus* st;
    uint32_t copies;            // variants that get these labels (equal minpts)
    const EpsParams* ep;        // reach pattern of the grid
};
// Clustering on grids whose cells are cliques: all minpts of one epsilon
// (slots), up to kSlots at a time.
constexpr int kSlots = 8;
struct CellArgs {
    uint32_t n;
    const uint32_t* deg;
    const uint32_t* gpos;
    const uint32_t* gorig;
    const uint32_t* gkey;
    const float2* glocal;       // FP32 coordinates relative to the own cell's origin
    const double2* gxy;         // FP64 coordinates, cell order
    const MpbBox* gbox;         // multiple-point box of each cell-ordered point
    GridParams g;
    const EpsParams* ep;
    const uint32_t* cell_start;
    const uint32_t* crow;       // sparse grids: row directory (see cell_row_range)
    const uint32_t* ccx;        // column of every non-empty cell
    uint2* crng;                // [2*rho+1][n] neighbour cells per row
    const uint32_t* clist;      // first point of every non-empty cell (ncl+1 entries)
    const uint32_t* ncl;        // device scalar
    const uint32_t* cscan;      // cell of point k: cscan[k + 1] - 1
    unsigned long long* cbest;  // per cell: largest degree and a point that has it (n entries)
    int m;                      // slots
    uint32_t mp[kSlots];        // minpts (0xffffffff: no cores)
    uint32_t copies[kSlots];    // variants that get the slot's labels
    // nested-epsilon reuse: comp_prev[v][pos] = component (its cluster start)
    // of the core at visit position pos in a variant with a larger or equal
    // epsilon and a smaller or equal minpts (nullptr: none); cores of
    // different components there cannot be connected here.  comp_out[v]
    // receives this slot's (nullptr: not kept).
    const uint32_t* comp_prev[kSlots];
    uint32_t* comp_out[kSlots];
    uint32_t* labels[kSlots];   // n labels in input order
    uint32_t* parent;           // [m][n] union-find over cells
    uint32_t* seed;             // [m][n] per root: min visit position of its cores
    uint32_t* cst;              // [m][n] per cell: start of its cores' cluster
    uint32_t* bits;             // [m][nw] visit positions at which clusters start
    uint32_t* brank;            // [m][nw] starts before each word
    uint32_t nw;                // start_words(n)
    const AsymPair* asym;
    const uint32_t* asym_count;
    uint32_t asym_cap;
    DeviceStatus* st;
};
// Words of the start bits of n visit positions (whole 32-byte groups).
inline uint32_t start_words(uint32_t n) { return ((n + 31u) / 32u + 7u) & ~7u; }
// nrows: 2*rho+1; row_cells: cells of a row within reach of a cell, at most;
// one_way: the table has one-way pairs; resolve_ws: m * resolve_scratch_bytes()
void launch_cells(const CellArgs& a, int nrows, int row_cells, bool one_way, void* resolve_ws,
                  cudaStream_t s);
size_t resolve_scratch_bytes();
// comp[gpos[k]] = seed of the component of core k, kNone for other points
// (after launch_uf_finish)
void launch_save_components(const ClusterArgs& a, uint32_t* comp, cudaStream_t s);

// Graph replay (vdb_options.graph).  A checkpoint re-checks device values
// that the host read while recording the call: each condition compares one
// value with what the host planned for (kGcLe64 / kGcLe32: at most a, and
// kGcLe64 adds the value to *sum when sum is set; kGcMask32: (value & a) == b;
// kGcGeF64 / kGcLeF64: a double at least / at most the double whose bits are
// a).  If all hold and no earlier checkpoint
// failed the conditional node after it runs; otherwise *bad = index (first
// failure) and the rest of the replay is skipped.
enum : uint32_t { kGcLe64 = 1, kGcLe32 = 2, kGcMask32 = 3, kGcGeF64 = 4, kGcLeF64 = 5 };
constexpr int kGraphConds = 8;
struct GraphCond {
    const void* ptr;
    unsigned long long* sum;
    unsigned long long a, b;
    uint32_t kind;
    uint32_t pad;
};
struct GraphCheck {
    GraphCond c[kGraphConds];
    int n;
    uint32_t index;  // 1-based checkpoint number
};
void launch_graph_check(const GraphCheck& chk, uint32_t* bad, cudaGraphConditionalHandle next,
                        cudaStream_t s);
// ---------------------------------------------------- clustering over points
void launch_uf_init(const ClusterArgs& a, bool fresh, cudaStream_t s);
void launch_uf_union(const ClusterArgs& a, int nblocks, cudaStream_t s);
void launch_uf_finish(const ClusterArgs& a, void* resolve_ws, cudaStream_t s);
void launch_border_and_write(const ClusterArgs& a, int nblocks, cudaStream_t s);
// the two halves of launch_border_and_write: border pull over rows
// [row_lo, row_hi) of the table held in nbr (from off_base), then the
// one-way in-edges and the label write (after every row has been pulled)
void launch_border_pull(const ClusterArgs& a, int nblocks, cudaStream_t s);
void launch_label_write(const ClusterArgs& a, cudaStream_t s);

}  // namespace vdb
