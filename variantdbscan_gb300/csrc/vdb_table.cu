// Epsilon-neighbourhood kernels: the count pass (|N_eps(p)| for every point,
// plus a bitmap of every candidate test) and the table pass (CSR neighbour
// table written from that bitmap).
//
// Work is split into units: a tile is up to 64 consecutive cell-ordered points
// (32 in small inputs) of one group of cells; its candidates are the points of the cells within reach in the
// rows cy-rho..cy+rho, i.e. 2*rho+1 contiguous ranges of the cell-ordered
// arrays; a unit is one tile and one chunk of unit_words*32 of its
// candidates.  Persistent warps take units from a global counter; each warp
// holds one tile's queries and stages its candidates in its own slice of shared
// memory.  Tiles of more than kLaneCand queries are tested lane = query (lane l:
// queries l and l+32), the others and all FP64 tests lane = candidate, and
// tiles of a few queries and candidates by a thread per point.  Tiles of
// thousands of candidates first compare the candidates' boxes, word by word.
//
// The neighbour predicate is the reference's (src/DBScan.cpp:665-702 with the
// R-tree candidate rule of src/RTree.h:1613-1625):
//   q in N(p)  <=>  sqrt(fl(fl(dx*dx)+fl(dy*dy))) <= eps     (dx = fl(px-qx), FP64)
//                   and q's multiple-point box overlaps [p-eps, p+eps]^2.
// sqrt is monotone and correctly rounded, so the first part is d2 <= thr with
// thr the largest double whose square root is <= eps.  The box part can only
// fail when d2 > tbox (a pair that deep inside the circle lies inside the query
// box).  Mixed precision: an FP32 quadratic form on cell-relative coordinates
// classifies a pair as in, out or within an error band around eps^2 whose
// width the host derives from the FP32 rounding bounds; only band pairs are
// re-tested with the FP64 predicate above, so membership is that of FP64.
//
// Table pass: the count pass stores, per tile, one 32-bit word per query and
// per 32 consecutive candidates (bit j: candidate j is a neighbour), laid out
// [word][query] so that a warp's 32 queries store 128 contiguous bytes.  The
// table pass turns each word into table entries (lane = bit), in candidate
// order: rows of 32-bit entries come out sorted, rows of 16-bit entries unit
// after unit, within a unit first the words that were expanded, then the runs
// of words that are neighbours as a whole.  An entry is 16 bits (the neighbour's
// position within its work unit of 512 to 4096 candidates; readers decode it
// through the tile's row segments and the count pass's per-unit counts) or 32 bits (the
// cell-ordered index).  Entries accepted in one direction only are flagged
// afterwards from the asymmetric-pair list.  When the bitmap does not fit in
// device memory, the fill kernel (blocks of kTT threads, kQPT queries a thread)
// re-tests the candidates and writes the table directly.
#include "vdb_lookback.cuh"

namespace vdb {

namespace {

constexpr int kTT = 256;              // threads per block
constexpr int kQPT = 2;               // queries per thread
constexpr int kChunk = 1024;          // candidates staged per round
constexpr unsigned kFull = 0xffffffffu;

// Row i (offset dy = i - rho) of the tile whose group starts at cell (cy, cx0):
// the candidate range [*st, *st + *len) and the key of the group's first cell
// in that row (so that key - base is the candidate's cell offset in x).
// Tile t's ranges come from a.trow_s / a.trow_e when those hold them (sparse
// grids, filled by the tile-words pass), else from the cell index.
__device__ __forceinline__ void tile_row(const TableArgs& a, const EpsParams* __restrict__ ep,
                                         int rho, uint32_t cy, uint32_t cx0, int i,
                                         uint32_t* st, uint32_t* len, uint32_t* base,
                                         uint32_t t = 0xffffffffu) {
    const int ry = (int)cy + i - rho;
    *st = 0;
    *len = 0;
    *base = 0;
    if (ry < 0 || ry >= (int)a.g.ncy) return;
    const int reach = ep->reach[i];
    const int lo_c = max((int)cx0 - reach, 0);
    const int hi_c = min((int)(cx0 + a.g.G - 1) + reach, (int)a.g.ncx - 1);
    const uint32_t rb = (uint32_t)ry * a.g.ncx_pad;
    uint32_t s = 0, e = 0;
    if (t != 0xffffffffu && a.trow_s) {
        const unsigned long long k = (unsigned long long)t * (uint32_t)(2 * rho + 1) + (uint32_t)i;
        s = a.trow_s[k];
        e = a.trow_e[k];
    } else {
        cell_row_range(a.g, a.cell_start, a.crow, a.ccx, a.clist, (uint32_t)ry, (uint32_t)lo_c,
                       (uint32_t)hi_c, &s, &e);
    }
    if (VDB_GUARD(a.st, s <= e && e <= a.n, 2, ((unsigned long long)s << 32) | e)) {
        *st = s;
        *len = e - s;
    }
    *base = rb + cx0;
}

// Cell-ordered index of candidate g of the tile (segments in shared memory).
__device__ __forceinline__ uint32_t tile_candidate(const uint32_t* s_seg_start,
                                                   const uint32_t* s_seg_off, int nrows,
                                                   uint32_t g, int* row) {
    int i = 0;
    while (i < nrows - 1 && s_seg_off[i + 1] <= g) i++;
    *row = i;
    return s_seg_start[i] + (g - s_seg_off[i]);
}

// Packed FP32 pairs (Blackwell f32x2 arithmetic): element-wise IEEE
// round-to-nearest, the same results as __fsub_rn / __fmaf_rn.
__device__ __forceinline__ unsigned long long f2_pack(float lo, float hi) {
    return ((unsigned long long)__float_as_uint(hi) << 32) | __float_as_uint(lo);
}
__device__ __forceinline__ unsigned long long f2_sub(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long f2_fma(unsigned long long a, unsigned long long b,
                                                     unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// ------------------------------------------------------ warp-granular kernels
// The count and table passes give every warp its own tile of at most kWQ
// queries (one group of cells): the warp stages its candidates in its own
// slice of shared memory and synchronises with __syncwarp only, so small
// tiles (the common case with cells of eps/2) keep every warp busy.

constexpr int kWPB = 8;               // warps per block
constexpr int kWQ = 64;               // queries per warp tile (lane l: queries l and l+32)
constexpr int kWC = 128;              // candidates staged per warp round
constexpr int kWXW = 16;              // bitmap words per round of the table pass
constexpr int kRQ = 128;              // band pairs queued per warp for FP64 re-tests

struct WarpRows {
    uint32_t start[kMaxRows];
    uint32_t off[kMaxRows + 1];
    uint32_t base[kMaxRows];
    float dyw[kMaxRows];
};

// Row segments of the tile whose group starts at cell (cy, cx0), prefix of
// their lengths in r.off (r.off[nrows] = number of candidates).
__device__ __forceinline__ void warp_rows(const TableArgs& a, const EpsParams* __restrict__ ep,
                                          int rho, int nrows, uint32_t cy, uint32_t cx0,
                                          float wf, WarpRows& r, int lane, uint32_t t) {
    for (int i = lane; i < nrows; i += 32) {
        uint32_t st, len, base;
        tile_row(a, ep, rho, cy, cx0, i, &st, &len, &base, t);
        r.start[i] = st;
        r.off[i + 1] = len;
        r.base[i] = base;
        r.dyw[i] = __fmul_rn((float)(i - rho), wf);
    }
    __syncwarp();
    if (lane == 0) {
        uint32_t acc = 0;
        r.off[0] = 0;
        for (int i = 0; i < nrows; i++) {
            acc += r.off[i + 1];
            r.off[i + 1] = acc;
        }
    }
    __syncwarp();
}

__device__ __forceinline__ float warp_min(float v) {
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float warp_max(float v) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// Records a pair accepted in one direction only (once per pair: kp < kq).
__device__ __forceinline__ void record_one_way(const TableArgs& a, uint32_t kp, uint32_t kq,
                                               uint32_t r) {
    if ((r != 1u && r != 2u) || kp >= kq) return;
    const uint32_t slot = atomicAdd(a.asym_n, 1u);
    if (slot < a.asym_cap) {
        AsymPair ap;
        ap.a = kp;
        ap.b = kq;
        ap.dir = r;
        ap.pad = 0u;
        a.asym[slot] = ap;
    } else {
        atomicOr(&a.st->flags, kStatAsymOverflow);
    }
}

// Tiles of at most kLaneCand queries are tested lane = candidate (a step per
// query) instead of lane = query (a step per candidate pair): a step costs
// about the same either way, so the lanes that a small tile leaves empty cost
// more than they test.  FP64 tests always go lane = candidate: they are bound
// by the FP64 pipe (2 lanes per cycle and SM), and only the last word of a
// tile has idle lanes.
constexpr uint32_t kLaneCand = 16;
// Word boxes.  A run of points that are next to each other in the cell order
// lies in a small box where the data are dense (points of a cell are ordered
// by subcell).  box[i] bounds the points [4i, 4i + 36), relative to the cell
// origin of point 4i, so it covers the 32 candidates of any word that starts
// at points 4i..4i+3; x0 > x1 when the run spans two grid rows, or more than
// kBoxCells cells of one (an edge far from point 4i is rounded at that distance:
// see box_pad).  Tiles of at least kBoxCand candidates compare each word's box
// with their queries' first: a box wholly inside or outside eps settles 64 x 32
// pairs without a test.
constexpr uint32_t kBoxCand = 2048;
constexpr uint32_t kBoxRun = 36;
constexpr uint32_t kBoxCells = 16;
// How far a box's edges are moved out along x and y in a tile of G cells with
// reach r in its own row (the largest): more than what the roundings can have
// moved them in.  With u = 2^-24, cells of width w and |positions| in the tile
// at most R = (G + r + 1) w, a point's stored x is off by at most
// u (kBoxCells + 1) w; the shift into the tile's coordinates, the pad's own
// subtraction and the candidate's coordinate that the box has to contain add at
// most u R each (an edge further out than R is one of a point between the run's
// first and the word's: rounding is monotone, it is no further in than the
// word's own).  Together u w (kBoxCells + 1 + 3 (G + r + 1)), against a pad of
// u w 16 (G + 2 r + 4), which is larger for all G, r >= 1.
__device__ __forceinline__ float box_pad(float wf, uint32_t G, int r) {
    static_assert(kBoxCells + 1 + 3 * (1 + 1 + 1) <= 16 * (1 + 2 + 4), "the pad covers the roundings");
    return 0x1p-20f * wf * (float)((int)G + 2 * r + 4);
}
__device__ __forceinline__ void word_box(const TableArgs& a, uint32_t i) {
    const uint32_t k0 = 4u * i;
    if (k0 >= a.n) return;
    const uint32_t key0 = a.gkey[k0], cy0 = key0 / a.g.ncx_pad;
    const uint32_t e = min(k0 + kBoxRun, a.n);
    const float wf = a.ep->wf;
    float4 b = make_float4(INFINITY, -INFINITY, INFINITY, -INFINITY);
    const uint32_t key1 = a.gkey[e - 1];
    if (key1 - key0 <= kBoxCells && key1 / a.g.ncx_pad == cy0) {
        for (uint32_t k = k0; k < e; k++) {
            const float2 loc = a.glocal[k];
            const float x = __fmaf_rn((float)(a.gkey[k] - key0), wf, loc.x);
            b.x = fminf(b.x, x);
            b.y = fmaxf(b.y, x);
            b.z = fminf(b.z, loc.y);
            b.w = fmaxf(b.w, loc.y);
        }
    }
    a.wbox[i] = b;
}

// Tiles of few queries and candidates are not worth a warp: its chain of
// dependent loads (unit, tile, segments, candidates) is the same for a tile of
// one query as for 64.  They are counted and expanded by a thread per point
// instead, which keeps 32 such chains in flight per warp.  Up to kSmallCand
// candidates the thread's serial tests stay shorter than that chain (1M
// uniform points, 3 epsilons: count 2,385 -> 310 us, expand 2,510 -> 65 us).
constexpr uint32_t kSmallCand = 128;
constexpr uint32_t kSmallQueries = 8;
// FP64 tests: only up to one word of candidates, and never fused.  A warp with
// lane = candidate keeps the FP64 pipe as busy as threads of unequal lists do
// (100k-point sweep: 2.8 ms against 3.1 with 128, 3.7 fused).
constexpr uint32_t kSmallCand64 = 32;
// Inputs of at most so many points: the first blocks of the count and expand
// kernels take the small tiles before they join the others (a launch of their
// own would add its whole latency, 15 to 30 us, to calls of 300).  Larger ones
// get a kernel of their own, at twice the warps per SM.
constexpr uint32_t kSmallFused = 1u << 17;

// Count pass of point k of a small tile: FP32 tests on coordinates relative to
// the point's own cell (FP64 inside the band, or for every pair), candidates
// in the tile's order, the loads of four at a time.  A block's threads take
// consecutive points.
template <bool MIXED>
__device__ void small_count(const TableArgs& a, uint32_t k) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t t = 0;
    bool mine = false;
    if (k < a.n) {
        t = a.ptile[k];
        mine = a.tile_uoff[t + 1] == a.tile_uoff[t];
    }
    if (!__any_sync(kFull, mine)) return;
    uint32_t cnt = 0, retest = 0, g = 0;
    if (mine) {
        const EpsParams* __restrict__ ep = a.ep;
        const ExactBounds xb = ep->xb;
        const float lo = ep->lo32, hi = ep->hi32, wf = a.ep->wf;
        const int rho = ep->rho, nrows = 2 * rho + 1;
        const uint32_t qs = a.tiles[t], Q = a.tiles[t + 1] - qs;
        const uint32_t key = a.gkey[k];
        const uint32_t key0 = a.gkey[qs], cy = key0 / a.g.ncx_pad;
        const uint32_t cx0 = (key0 - cy * a.g.ncx_pad) / a.g.G * a.g.G;
        const float2 q = a.glocal[k];
        uint32_t* const bm = a.bitmap ? a.bitmap + a.tile_boff[t] + (k - qs) : nullptr;
        uint32_t word = 0;
        for (int i = 0; i < nrows; i++) {
            uint32_t st, len, base;
            tile_row(a, ep, rho, cy, cx0, i, &st, &len, &base, t);
            const uint32_t own = key + (uint32_t)((i - rho) * (int)a.g.ncx_pad);
            const float dyw = __fmul_rn((float)(i - rho), wf);
            for (uint32_t j0 = st; j0 < st + len; j0 += 32) {
                const uint32_t m = min(32u, st + len - j0);
                uint32_t in = 0, band = MIXED ? 0u : (m == 32u ? kFull : (1u << m) - 1u);
                if (MIXED) {
                    for (uint32_t b0 = 0; b0 < m; b0 += 4) {
                        float2 c[4];
                        uint32_t ck[4];
#pragma unroll
                        for (uint32_t b = 0; b < 4; b++) {
                            const uint32_t j = j0 + min(b0 + b, m - 1u);
                            c[b] = a.glocal[j];
                            ck[b] = a.gkey[j];
                        }
#pragma unroll
                        for (uint32_t b = 0; b < 4; b++) {
                            const float dx =
                                __fsub_rn(q.x, __fmaf_rn((float)(int)(ck[b] - own), wf, c[b].x));
                            const float dy = __fsub_rn(q.y, __fadd_rn(c[b].y, dyw));
                            const float d2 = __fmaf_rn(dx, dx, __fmul_rn(dy, dy));
                            if (b0 + b < m) {
                                if (d2 < lo) in |= 1u << (b0 + b);
                                else if (d2 <= hi) band |= 1u << (b0 + b);
                            }
                        }
                    }
                }
                // (the lanes' re-tests run side by side)
                for (; band; band &= band - 1u) {
                    const uint32_t b = (uint32_t)__ffs(band) - 1u, j = j0 + b;
                    const uint32_t r = exact_pair(a.gxy[k], a.gxy[j], k, j, xb, a.gbox);
                    retest += MIXED ? 1u : 0u;
                    if (r & 1u) in |= 1u << b;
                    record_one_way(a, k, j, r);
                }
                cnt += (uint32_t)__popc(in);
                const uint32_t sh = g & 31u;
                word |= in << sh;
                if (sh + m >= 32u) {
                    if (bm) bm[(unsigned long long)(g >> 5) * Q] = word;
                    word = sh ? in >> (32u - sh) : 0u;
                }
                g += m;
            }
        }
        if ((g & 31u) && bm) bm[(unsigned long long)(g >> 5) * Q] = word;
        a.deg[k] = cnt;
    }
    const uint32_t tests = __reduce_add_sync(kFull, g), again = __reduce_add_sync(kFull, retest);
    const uint32_t pairs = __reduce_add_sync(kFull, cnt);
    if (lane == 0) {
        atomicAdd(&a.st->candidates, (unsigned long long)tests);
        if (again) atomicAdd(&a.st->retested, (unsigned long long)again);
        if (a.pair_sum) atomicAdd(a.pair_sum, (unsigned long long)pairs);
    }
}

template <bool MIXED>
__global__ void __launch_bounds__(kTT) small_count_kernel(TableArgs a) {
    pdl_sync();
    small_count<MIXED>(a, blockIdx.x * blockDim.x + threadIdx.x);
}

// Table row of point k of a small tile.
template <typename E>
__device__ void small_expand(const TableArgs& a, uint32_t k) {
    const uint32_t t = a.ptile[k];
    if (a.tile_uoff[t + 1] != a.tile_uoff[t]) return;
    const uint32_t qs = a.tiles[t], Q = a.tiles[t + 1] - qs;
    const uint32_t* __restrict__ bm = a.bitmap + a.tile_boff[t] + (k - qs);
    E* dst = reinterpret_cast<E*>(a.nbr) + (a.off[k] - a.off_base);
    E* const end = reinterpret_cast<E*>(a.nbr) + (a.off[k + 1] - a.off_base);
    const int rho = a.ep->rho, nrows = 2 * rho + 1;
    const uint32_t key0 = a.gkey[qs], cy = key0 / a.g.ncx_pad;
    const uint32_t cx0 = (key0 - cy * a.g.ncx_pad) / a.g.G * a.g.G;
    // 32-bit entries: the segment that holds the position
    int row = -1;
    uint32_t st = 0, before = 0, after = 0;
    for (uint32_t w = 0; dst < end && w < kSmallCand / 32; w++) {
        for (uint32_t m = bm[(unsigned long long)w * Q]; m && dst < end; m &= m - 1u) {
            const uint32_t g = w * 32u + (uint32_t)__ffs(m) - 1u;
            if (sizeof(E) == 2) {
                *dst++ = (E)g;
            } else {
                while (g >= after && row + 1 < nrows) {
                    uint32_t len, base;
                    before = after;
                    tile_row(a, a.ep, rho, cy, cx0, ++row, &st, &len, &base, t);
                    after = before + len;
                }
                *dst++ = (E)(st + (g - before));
            }
        }
    }
}

template <typename E>
__global__ void __launch_bounds__(kTT) small_expand_kernel(TableArgs a) {
    pdl_sync();
    const uint32_t k = a.row_lo + blockIdx.x * blockDim.x + threadIdx.x;
    if (k < a.row_hi) small_expand<E>(a, k);
}

// Count pass over work units (tile, chunk of unit_words*32 candidates): adds
// each query's neighbours in the chunk to deg, records them in parts (for the
// table pass) and, when a.bitmap is set, stores the chunk's test bitmap
// ([word][query] words; bit j of word w: candidate 32w+j is a neighbour).
template <bool MIXED>
__global__ void __launch_bounds__(kWPB * 32, 3) count_kernel(TableArgs a) {
    pdl_sync();
    __shared__ WarpRows s_rows[kWPB];
    __shared__ uint32_t s_id[kWPB][MIXED ? kWC : 1];
    // lane = query: candidate pairs (x_a, x_b, y_a, y_b); lane = candidate:
    // queries (x, y, (L - |q|^2)/2)
    __shared__ float4 s_relp[kWPB][MIXED ? kWC / 2 : 1];
    __shared__ float2 s_hcp[kWPB][MIXED ? kWC / 2 : 1];
    // band pairs of a word are re-tested in FP64 32 at a time, whatever query
    // they belong to: queue of (query slot, candidate) entries, the queries'
    // FP64 coordinates and the accepted bits per query slot
    __shared__ uint16_t s_rq[kWPB][MIXED ? kRQ : 1];
    __shared__ double2 s_qd[kWPB][kWQ];
    __shared__ uint32_t s_madd[kWPB][MIXED ? kWQ : 1];
    static_assert(kWC / 2 >= kWQ, "queries fit the candidate pairs' array");

    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    WarpRows& rows = s_rows[wib];
    double2* sqd = s_qd[wib];
    const EpsParams* __restrict__ ep = a.ep;
    const ExactBounds xb = ep->xb;
    const float L = ep->L32, wq = ep->w32;
    const int rho = ep->rho;
    const int nrows = 2 * rho + 1;
    const float wf = a.ep->wf;
    const uint32_t nunits = *a.nunits;
    const uint32_t ncx_pad = a.g.ncx_pad, G = a.g.G;
    const float fnan = __int_as_float(0x7fc00000);
    const double dnan = __longlong_as_double(0x7ff8000000000000ll);
    unsigned long long my_retest = 0, my_pairs = 0;
    if (MIXED) {
        s_madd[wib][lane] = 0u;
        s_madd[wib][lane + 32] = 0u;
    }

    if (MIXED && a.n <= kSmallFused)
        for (uint32_t k0 = blockIdx.x * (kWPB * 32u); k0 < a.n; k0 += gridDim.x * (kWPB * 32u))
            small_count<MIXED>(a, k0 + threadIdx.x);

    for (;;) {
        uint32_t u = 0;
        if (lane == 0) u = atomicAdd(a.tile_counter, 1u);
        u = __shfl_sync(kFull, u, 0);
        if (u >= nunits) break;
        const uint32_t t = a.ulist[u];
        const uint32_t chunk = u - a.tile_uoff[t];
        const uint32_t qs = a.tiles[t], qe = a.tiles[t + 1];
        if (!(qs < qe && qe <= a.n && qe - qs <= kUnitQ)) {
            if (lane == 0) guard_fail(a.st, 1, ((unsigned long long)qs << 32) | qe);
            continue;
        }
        const uint32_t Q = qe - qs;
        const uint32_t key0 = a.gkey[qs];
        const uint32_t cy = key0 / ncx_pad;
        const uint32_t cx0 = (key0 - cy * ncx_pad) / G * G;
        const uint32_t tile_base = cy * ncx_pad + cx0;
        warp_rows(a, ep, rho, nrows, cy, cx0, wf, rows, lane, t);
        const uint32_t C = rows.off[nrows];
        const uint32_t cbeg = chunk * a.unit_words * 32u;
        const uint32_t cend = min(C, cbeg + a.unit_words * 32u);
        if (cbeg >= cend) continue;
        if (lane == 0) atomicAdd(&a.st->candidates, (unsigned long long)(cend - cbeg) * Q);
        const unsigned long long bm0 = a.bitmap ? a.tile_boff[t] : 0ull;

        float qx[2], qy[2];
        uint32_t cnt[2] = {0u, 0u};
        const uint32_t qk[2] = {qs + (uint32_t)lane, qs + (uint32_t)lane + 32u};
#pragma unroll
        for (int q = 0; q < 2; q++) {
            double2 qd = make_double2(dnan, dnan);
            qx[q] = qy[q] = fnan;
            if (qk[q] < qe) {
                if (MIXED) {
                    const float2 loc = a.glocal[qk[q]];
                    const int dcx = (int)(a.gkey[qk[q]] - tile_base);
                    qx[q] = __fmaf_rn((float)dcx, wf, loc.x);
                    qy[q] = loc.y;
                }
                qd = a.gxy[qk[q]];
            }
            sqd[lane + 32 * q] = qd;
        }
        const bool two = Q > 32;  // second query slot used by some lane
        bool settled = false;     // the unit's words settled by their boxes have been recorded
        // the float above w (w > 0)
        const float wup = __uint_as_float(__float_as_uint(wq) + 1u);
        const unsigned long long w2p = f2_pack(wup, wup);

        if (!MIXED) {
            __syncwarp();
            for (uint32_t cb = cbeg; cb < cend; cb += 32) {
                uint32_t k = 0;
                int i;
                double2 cd = make_double2(dnan, dnan);
                if (cb + (uint32_t)lane < cend) {
                    k = tile_candidate(rows.start, rows.off, nrows, cb + (uint32_t)lane, &i);
                    if (VDB_GUARD(a.st, k < a.n, 3, k)) cd = a.gxy[k];
                }
                uint32_t w[2] = {0u, 0u};
                auto step = [&](uint32_t q, uint32_t* word) {
                    // d2 is >= +0 or NaN; compared as ordered integers
                    // (ExactBounds), NaN by its bits above those of infinity
                    const double2 qd = sqd[q];
                    const double dx = __dsub_rn(qd.x, cd.x), dy = __dsub_rn(qd.y, cd.y);
                    const long long d2b =
                        __double_as_longlong(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)));
                    const bool num = (unsigned long long)d2b <= 0x7ff0000000000000ull;
                    bool in = num && d2b <= xb.tbox;
                    const bool band = num && !in && d2b <= xb.thr;
                    if (__any_sync(kFull, band)) {
                        if (band) {
                            const uint32_t r = exact_pair(qd, cd, qs + q, k, xb, a.gbox);
                            my_retest++;
                            in = (r & 1u) != 0u;
                            record_one_way(a, qs + q, k, r);
                        }
                    }
                    const uint32_t m = __ballot_sync(kFull, in);
                    if ((uint32_t)lane == (q & 31u)) *word = m;
                };
                for (uint32_t q = 0; q < min(Q, 32u); q++) step(q, &w[0]);
                for (uint32_t q = 32; q < Q; q++) step(q, &w[1]);
                const unsigned long long wrow = bm0 + (unsigned long long)(cb >> 5) * Q;
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    if (qk[q] < qe) {
                        cnt[q] += __popc(w[q]);
                        if (a.bitmap) a.bitmap[wrow + (qk[q] - qs)] = w[q];
                    }
                }
            }
            __syncwarp();
        } else if (Q <= kLaneCand) {
            float4* sq = s_relp[wib];
            uint16_t* rq = s_rq[wib];
            uint32_t* madd = s_madd[wib];
            uint32_t* ids = s_id[wib];
            static_assert(kLaneCand * 4 <= kWQ, "the accepted bits' words");
            if ((uint32_t)lane < Q) {
                const float q2 = __fmaf_rn(qx[0], qx[0], __fmul_rn(qy[0], qy[0]));
                sq[lane] = make_float4(qx[0], qy[0], -0.5f * __fsub_rn(q2, L), 0.f);
            }
            __syncwarp();
            for (uint32_t cb = cbeg; cb < cend; cb += kWC) {
                // this lane's four candidates (words s = 0..3)
                __syncwarp();  // (ids of the candidates before have been read)
                unsigned long long X[2], Y[2], H[2];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    float rx[2], ry[2], hc[2];
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const uint32_t g = cb + 32u * (2 * h + e) + (uint32_t)lane;
                        rx[e] = ry[e] = hc[e] = fnan;
                        uint32_t id = 0;
                        if (g < cend) {
                            int i;
                            const uint32_t k = tile_candidate(rows.start, rows.off, nrows, g, &i);
                            if (VDB_GUARD(a.st, k < a.n, 3, k)) {
                                const float2 loc = a.glocal[k];
                                const int dcx = (int)(a.gkey[k] - rows.base[i]);
                                rx[e] = __fmaf_rn((float)dcx, wf, loc.x);
                                ry[e] = __fadd_rn(loc.y, rows.dyw[i]);
                                hc[e] = 0.5f * __fmaf_rn(rx[e], rx[e], __fmul_rn(ry[e], ry[e]));
                                id = k;
                            }
                        }
                        ids[32 * (2 * h + e) + lane] = id;
                    }
                    X[h] = f2_pack(rx[0], rx[1]);
                    Y[h] = f2_pack(ry[0], ry[1]);
                    H[h] = f2_pack(hc[0], hc[1]);
                }
                const uint32_t nwv = (min((uint32_t)kWC, cend - cb) + 31u) >> 5;
                uint32_t w[4] = {0u, 0u, 0u, 0u}, amb[4] = {0u, 0u, 0u, 0u};
                for (uint32_t q = 0; q < Q; q++) {
                    const float4 Qv = sq[q];
                    const unsigned long long qxx = f2_pack(Qv.x, Qv.x), qyy = f2_pack(Qv.y, Qv.y),
                                             nh = f2_pack(Qv.z, Qv.z);
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        if (h == 1 && nwv <= 2) break;
                        // the filter of the lane = query form below, two words at a time
                        const unsigned long long s =
                            f2_sub(H[h], f2_fma(qxx, X[h], f2_fma(qyy, Y[h], nh)));
                        const unsigned long long nwm = f2_sub(s, w2p);
                        const bool in0 = (int)(uint32_t)s < 0, in1 = (int)(uint32_t)(s >> 32) < 0;
                        const bool b0 = !in0 && (int)(uint32_t)nwm < 0;
                        const bool b1 = !in1 && (int)(uint32_t)(nwm >> 32) < 0;
                        const uint32_t m0 = __ballot_sync(kFull, in0), m1 = __ballot_sync(kFull, in1);
                        if ((uint32_t)lane == q) {
                            w[2 * h] = m0;
                            w[2 * h + 1] = m1;
                        }
                        if (__any_sync(kFull, b0 || b1)) {
                            const uint32_t a0 = __ballot_sync(kFull, b0), a1 = __ballot_sync(kFull, b1);
                            if ((uint32_t)lane == q) {
                                amb[2 * h] = a0;
                                amb[2 * h + 1] = a1;
                            }
                        }
                    }
                }
                // pairs in the band, queued as below (entries: query, candidate)
                if (__any_sync(kFull, (amb[0] | amb[1] | amb[2] | amb[3]) != 0u)) {
                    const uint32_t c =
                        __popc(amb[0]) + __popc(amb[1]) + __popc(amb[2]) + __popc(amb[3]);
                    uint32_t incl = c;
#pragma unroll
                    for (int d = 1; d < 32; d <<= 1) {
                        const uint32_t v = __shfl_up_sync(kFull, incl, d);
                        if (lane >= d) incl += v;
                    }
                    const uint32_t excl = incl - c, total = __shfl_sync(kFull, incl, 31);
                    for (uint32_t pb = 0; pb < total; pb += kRQ) {
                        uint32_t idx = excl;
#pragma unroll
                        for (int s = 0; s < 4; s++) {
                            for (uint32_t bits = amb[s]; bits; bits &= bits - 1u, idx++) {
                                if (idx >= pb && idx < pb + kRQ)
                                    rq[idx - pb] = (uint16_t)(((uint32_t)lane << 7) | (32u * s) |
                                                              (uint32_t)(__ffs(bits) - 1));
                            }
                        }
                        __syncwarp();
                        const uint32_t ne = min((uint32_t)kRQ, total - pb);
                        for (uint32_t e = lane; e < ne; e += 32) {
                            const uint32_t ent = rq[e], q = ent >> 7, jj = ent & 127u;
                            const uint32_t kq = ids[jj];
                            const uint32_t r =
                                exact_pair(sqd[q], a.gxy[kq], qs + q, kq, xb, a.gbox);
                            my_retest++;
                            if (r & 1u) atomicOr(&madd[q * 4 + (jj >> 5)], 1u << (jj & 31u));
                            record_one_way(a, qs + q, kq, r);
                        }
                        __syncwarp();
                    }
                    if ((uint32_t)lane < Q) {
#pragma unroll
                        for (int s = 0; s < 4; s++) {
                            w[s] |= madd[lane * 4 + s];
                            madd[lane * 4 + s] = 0u;
                        }
                    }
                    __syncwarp();
                }
                if ((uint32_t)lane < Q) {
                    const unsigned long long wrow = bm0 + (unsigned long long)(cb >> 5) * Q + (uint32_t)lane;
#pragma unroll
                    for (int s = 0; s < 4; s++) {
                        cnt[0] += __popc(w[s]);
                        if (a.bitmap && (uint32_t)s < nwv) a.bitmap[wrow + (unsigned long long)s * Q] = w[s];
                    }
                }
            }
            __syncwarp();
        } else {
            uint16_t* rq = s_rq[wib];
            uint32_t* madd = s_madd[wib];
            float4* relp = s_relp[wib];
            float2* hcp = s_hcp[wib];
            uint32_t* ids = s_id[wib];
            unsigned long long qxx[2], qyy[2], nhq2[2];
#pragma unroll
            for (int q = 0; q < 2; q++) {
                qxx[q] = f2_pack(qx[q], qx[q]);
                qyy[q] = f2_pack(qy[q], qy[q]);
                // -(|q|^2 - L)/2 (halving and negation are exact)
                const float q2 = __fmaf_rn(qx[q], qx[q], __fmul_rn(qy[q], qy[q]));
                const float nhq = -0.5f * __fsub_rn(q2, L);
                nhq2[q] = f2_pack(nhq, nhq);
            }
            const bool boxes = a.wbox && C >= kBoxCand;
            if (boxes) settled = true;
            float bx0 = 0.f, bx1 = 0.f, by0 = 0.f, by1 = 0.f;  // the queries' box (fmin/fmax skip NaN)
            float pad = 0.f;
            if (boxes) {
                bx0 = warp_min(fminf(qx[0], qx[1]));
                bx1 = warp_max(fmaxf(qx[0], qx[1]));
                by0 = warp_min(fminf(qy[0], qy[1]));
                by1 = warp_max(fmaxf(qy[0], qy[1]));
                pad = box_pad(wf, G, ep->reach[rho]);
            }

            // blocks of 32 words: lane l looks at word wb + l
            for (uint32_t wb = cbeg >> 5; wb * 32u < cend; wb += 32) {
                const uint32_t nwb = min(32u, ((cend + 31u) >> 5) - wb);
                uint32_t todo = nwb >= 32u ? kFull : (1u << nwb) - 1u;  // words to test
                if (boxes) {
                    bool in = false, out = false;
                    const uint32_t g0 = (wb + (uint32_t)lane) * 32u, g1 = min(g0 + 32u, cend);
                    if ((uint32_t)lane < nwb) {
                        int i;
                        const uint32_t k = tile_candidate(rows.start, rows.off, nrows, g0, &i);
                        if (g1 <= rows.off[i + 1] && VDB_GUARD(a.st, k < a.n, 3, k)) {
                            const float4 b = a.wbox[k >> 2];
                            if (b.x <= b.y) {
                                // The padded box holds the FP32 coordinates of
                                // the word's candidates.  Rounding is monotone:
                                // the largest |q - c| per axis, rounded, is at
                                // least every rounded |q - c|, and its FP32 d2
                                // at least every pair's; the smallest likewise.
                                // So d2max < lo32 (d2min > hi32) decides all
                                // pairs of the two boxes as their own FP32 d2
                                // would.
                                const float dcx = (float)(int)(a.gkey[k & ~3u] - rows.base[i]);
                                const float x0 = __fmaf_rn(dcx, wf, b.x) - pad;
                                const float x1 = __fmaf_rn(dcx, wf, b.y) + pad;
                                const float y0 = b.z + rows.dyw[i] - pad, y1 = b.w + rows.dyw[i] + pad;
                                const float mx = fmaxf(__fsub_rn(x1, bx0), __fsub_rn(bx1, x0));
                                const float my = fmaxf(__fsub_rn(y1, by0), __fsub_rn(by1, y0));
                                const float nx = fmaxf(fmaxf(__fsub_rn(x0, bx1), __fsub_rn(bx0, x1)), 0.f);
                                const float ny = fmaxf(fmaxf(__fsub_rn(y0, by1), __fsub_rn(by0, y1)), 0.f);
                                in = __fmaf_rn(mx, mx, __fmul_rn(my, my)) < ep->lo32;
                                out = __fmaf_rn(nx, nx, __fmul_rn(ny, ny)) > ep->hi32;
                            }
                        }
                    }
                    const uint32_t mi = __ballot_sync(kFull, in), mo = __ballot_sync(kFull, out);
                    todo &= ~(mi | mo);
                    if (a.wflags && lane == 0)
                        a.wflags[(unsigned long long)u * flag_blocks(a.unit_words) + (wb - (cbeg >> 5)) / 32u] =
                            make_uint2(mi, mo);
                    const uint32_t add = __reduce_add_sync(kFull, in ? g1 - g0 : 0u);
                    if (qk[0] < qe) cnt[0] += add;
                    if (qk[1] < qe) cnt[1] += add;
                    if (a.bitmap) {
                        for (uint32_t l = mi | mo; l; l &= l - 1u) {
                            const uint32_t w = (uint32_t)__ffs(l) - 1u, word = wb + w;
                            const uint32_t left = cend - word * 32u;
                            const uint32_t m = !((mi >> w) & 1u) ? 0u
                                               : left >= 32u     ? kFull
                                                                 : (1u << left) - 1u;
                            const unsigned long long wrow = bm0 + (unsigned long long)word * Q;
                            if (qk[0] < qe) a.bitmap[wrow + (qk[0] - qs)] = m;
                            if (qk[1] < qe) a.bitmap[wrow + (qk[1] - qs)] = m;
                        }
                    }
                }
                while (todo) {
                // the next (up to) four words
                uint32_t word[kWC / 32];
                uint32_t nst = 0;
#pragma unroll
                for (int s = 0; s < kWC / 32; s++) {
                    word[s] = 0xffffffffu;
                    if (todo) {
                        word[s] = wb + (uint32_t)__ffs(todo) - 1u;
                        todo &= todo - 1u;
                        nst = (uint32_t)s + 1u;
                    }
                }
#pragma unroll
                for (int s = 0; s < kWC / 32; s++) {
                    const uint32_t j = (uint32_t)lane + 32u * s;
                    const uint32_t cg = word[s] * 32u + (uint32_t)lane;
                    uint32_t k = 0;
                    float rx = fnan, ry = fnan;
                    if (word[s] != 0xffffffffu && cg < cend) {
                        int i;
                        k = tile_candidate(rows.start, rows.off, nrows, cg, &i);
                        if (VDB_GUARD(a.st, k < a.n, 3, k)) {
                            const float2 loc = a.glocal[k];
                            const int dcx = (int)(a.gkey[k] - rows.base[i]);
                            rx = __fmaf_rn((float)dcx, wf, loc.x);
                            ry = __fadd_rn(loc.y, rows.dyw[i]);
                        } else {
                            k = 0;
                        }
                    }
                    // pair slot of candidate j: (j>>5)*16 + (j&15), element j>>4 & 1
                    float* pslot = reinterpret_cast<float*>(&relp[(j >> 5) * 16 + (j & 15)]) +
                                   ((j >> 4) & 1);
                    float* hslot = reinterpret_cast<float*>(&hcp[(j >> 5) * 16 + (j & 15)]) +
                                   ((j >> 4) & 1);
                    pslot[0] = rx;
                    pslot[2] = ry;
                    hslot[0] = 0.5f * __fmaf_rn(rx, rx, __fmul_rn(ry, ry));
                    ids[j] = k;
                }
                __syncwarp();
#pragma unroll 1
                for (uint32_t j0 = 0; j0 < nst * 32u; j0 += 32) {
                    uint32_t m[2] = {0u, 0u}, amb[2] = {0u, 0u};
                    {
                        // Candidates jj and jj+16 are tested together with packed FP32
                        // pair instructions; sign bits are gathered by funnel shifts
                        // (bit 31-jj, reversed below).
                        // nS =|c|^2/2 - (q.c - (|q|^2 - L)/2) = (d2 - L)/2: two
                        // fma and one subtraction per test; its sign is the
                        // in-mask.  The sign of nS - w' (w' the float above w, so
                        // negative <=> nS <= w; a difference of floats is zero only
                        // for equal operands, so its sign is exact) marks the tests
                        // that are not out; band = not out and not in.  NaN (empty
                        // query or candidate slots) has both signs clear.
                        uint32_t ma[2] = {0u, 0u}, mb[2] = {0u, 0u}, oa[2] = {0u, 0u}, ob[2] = {0u, 0u};
                        const ulonglong2* pr = reinterpret_cast<const ulonglong2*>(relp) + (j0 >> 5) * 16;
                        const unsigned long long* ph =
                            reinterpret_cast<const unsigned long long*>(hcp) + (j0 >> 5) * 16;
#pragma unroll
                        for (int jj = 0; jj < 16; jj++) {
                            const ulonglong2 c = pr[jj];  // (x_a, x_b), (y_a, y_b)
                            const unsigned long long hc = ph[jj];  // (|c_a|^2/2, |c_b|^2/2)
#pragma unroll
                            for (int q = 0; q < 2; q++) {
                                if (q == 1 && !two) break;
                                const unsigned long long ay = f2_fma(qyy[q], c.y, nhq2[q]);
                                const unsigned long long qc = f2_fma(qxx[q], c.x, ay);
                                const unsigned long long s = f2_sub(hc, qc);
                                const unsigned long long nw = f2_sub(s, w2p);
                                ma[q] = __funnelshift_l((uint32_t)s, ma[q], 1);
                                mb[q] = __funnelshift_l((uint32_t)(s >> 32), mb[q], 1);
                                oa[q] = __funnelshift_l((uint32_t)nw, oa[q], 1);
                                ob[q] = __funnelshift_l((uint32_t)(nw >> 32), ob[q], 1);
                            }
                        }
#pragma unroll
                        for (int q = 0; q < 2; q++) {
                            m[q] = __brev((ma[q] << 16) | (mb[q] & 0xffffu));
                            amb[q] = __brev((oa[q] << 16) | (ob[q] & 0xffffu)) & ~m[q];
                        }
                        // pairs in the band: exact FP64 predicate, 32 pairs per step
                        // of the warp (queued in shared memory, whatever their query)
                        if (__any_sync(kFull, (amb[0] | amb[1]) != 0u)) {
                            const uint32_t c = __popc(amb[0]) + __popc(amb[1]);
                            uint32_t incl = c;
#pragma unroll
                            for (int d = 1; d < 32; d <<= 1) {
                                const uint32_t v = __shfl_up_sync(kFull, incl, d);
                                if (lane >= d) incl += v;
                            }
                            const uint32_t excl = incl - c;
                            const uint32_t total = __shfl_sync(kFull, incl, 31);
                            for (uint32_t pb = 0; pb < total; pb += kRQ) {
                                uint32_t idx = excl;
#pragma unroll
                                for (int q = 0; q < 2; q++) {
                                    for (uint32_t bits = amb[q]; bits; bits &= bits - 1u, idx++) {
                                        if (idx >= pb && idx < pb + kRQ)
                                            rq[idx - pb] = (uint16_t)(((uint32_t)lane << 6) |
                                                                      ((uint32_t)q << 5) |
                                                                      (uint32_t)(__ffs(bits) - 1));
                                    }
                                }
                                __syncwarp();
                                const uint32_t ne = min((uint32_t)kRQ, total - pb);
                                for (uint32_t e = lane; e < ne; e += 32) {
                                    const uint32_t ent = rq[e];
                                    const uint32_t slot_q = (ent >> 6) + 32u * ((ent >> 5) & 1u);
                                    const uint32_t jj = ent & 31u;
                                    const uint32_t kp = qs + slot_q;
                                    const uint32_t kq = ids[j0 + jj];
                                    const uint32_t r =
                                        exact_pair(sqd[slot_q], a.gxy[kq], kp, kq, xb, a.gbox);
                                    my_retest++;
                                    if (r & 1u) atomicOr(&madd[slot_q], 1u << jj);
                                    record_one_way(a, kp, kq, r);
                                }
                                __syncwarp();
                            }
                            m[0] |= madd[lane];
                            m[1] |= madd[lane + 32];
                            madd[lane] = 0u;
                            madd[lane + 32] = 0u;
                            __syncwarp();
                        }
                    }
                    const uint32_t wj = j0 == 0 ? word[0] : j0 == 32 ? word[1] : j0 == 64 ? word[2] : word[3];
                    const unsigned long long wrow = bm0 + (unsigned long long)wj * Q;
#pragma unroll
                    for (int q = 0; q < 2; q++) {
                        if (qk[q] < qe) {
                            cnt[q] += __popc(m[q]);
                            if (a.bitmap) a.bitmap[wrow + (qk[q] - qs)] = m[q];
                        }
                    }
                }
                __syncwarp();
                }
            }
        }
        if (a.wflags && !settled && (uint32_t)lane < flag_blocks(a.unit_words))
            a.wflags[(unsigned long long)u * flag_blocks(a.unit_words) + lane] = make_uint2(0u, 0u);
#pragma unroll
        for (int q = 0; q < 2; q++) {
            if (qk[q] < qe) {
                if (cnt[q]) atomicAdd(&a.deg[qk[q]], cnt[q]);
                if (a.parts) a.parts[(unsigned long long)u * kUnitQ + lane + 32u * q] = cnt[q];
                my_pairs += cnt[q];
            }
        }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        my_retest += __shfl_down_sync(kFull, my_retest, d);
        my_pairs += __shfl_down_sync(kFull, my_pairs, d);
    }
    if (lane == 0 && my_retest) atomicAdd(&a.st->retested, my_retest);
    if (lane == 0 && my_pairs && a.pair_sum) atomicAdd(a.pair_sum, my_pairs);
}

// Table pass over the same work units: neighbour ids from the count pass's
// bitmap.  A unit's rows start at the row offsets plus the neighbours of the
// tile's earlier units (parts).  The warp expands the unit in rounds of kWXW
// words.  Each lane keeps the ids of its bit of the round's words in
// registers.  The round's words are transposed through the warp's shared
// memory, 32 queries at a time: lane q loads query q's words (coalesced over
// q), adds up their popcounts into the in-row offset of every word and takes
// its row cursor forward; every query's slot (words, offsets, cursor, count)
// is then read back with a few broadcast vector loads.  Lane l shifts each word
// left by 31-l: the sign bit is its own bit and the popcount is its rank among
// the word's neighbours plus one, so the entry goes to the word's staging
// address (that of the entry before its first) plus 4 * popcount.  Rows come
// out in candidate order, which is increasing neighbour index.
//
// Stores: a query's ids of a round are first placed in a shared-memory
// staging buffer (one store per word, lane = bit, at the same position modulo
// 16 bytes as their place in the table); the 16-byte-aligned middle of the
// segment then goes to the table as one asynchronous bulk copy, and the at
// most 3 + 3 entries before and after it as plain stores.  The warp's stores
// thus become shared-memory stores that do not wait on the memory system, and
// the copies run while the warp expands the next queries.  Two staging buffers
// per warp, used in turn: before a buffer is refilled, the copy last issued
// from it (if any) must have read it.
//
// A round writes a query's segment only up to its last 32-byte boundary; the
// at most 7 entries after it are kept in shared memory and staged again in
// front of the query's next round (the unit's last round writes everything).
// The row's next segment follows a whole round over the tile's other queries
// later, and a sector left half written for that long was measured to cost
// about a third of the write bandwidth.
constexpr int kXS = 36;  // words per query slot: 16 words, 16 staging addresses, cursor, counts
constexpr int kXPB = 3;        // warps per block

// Entry layout of a table with entries of type E (uint32_t: cell-ordered
// index; uint16_t: position in the tile's candidate list): entries per 16
// bytes (the bulk-copy granule) and per 32-byte sector (carry alignment), and
// staging entries per buffer (phase + carried entries + one round's entries,
// rounded up to a granule).
template <typename E>
struct XFmt {
    static constexpr uint32_t kVec = 16 / sizeof(E);
    static constexpr uint32_t kSec = 32 / sizeof(E);
    static constexpr uint32_t kStage = ((kVec - 1) + (kSec - 1) + kWXW * 32 + kVec - 1) / kVec * kVec;
};

// Stores v at shared-memory address addr if x is negative (one predicated store).
__device__ __forceinline__ void st_shared_if_neg(int x, uint32_t addr, uint32_t v) {
    asm volatile("{ .reg .pred p; setp.lt.s32 p, %0, 0; @p st.shared.u32 [%1], %2; }"
                 ::"r"(x), "r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void st_shared_if_neg(int x, uint32_t addr, uint16_t v) {
    asm volatile("{ .reg .pred p; setp.lt.s32 p, %0, 0; @p st.shared.u16 [%1], %2; }"
                 ::"r"(x), "r"(addr), "h"(v) : "memory");
}

__device__ __forceinline__ void bulk_copy_to_global(void* gdst, const void* ssrc,
                                                    uint32_t bytes) {
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(ssrc);
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
                 ::"l"(gdst), "r"(s), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

template <typename E>
__global__ void __launch_bounds__(kXPB * 32, 6) expand_kernel(TableArgs a) {
    pdl_sync();
    constexpr uint32_t kVec = XFmt<E>::kVec, kSec = XFmt<E>::kSec, kStage = XFmt<E>::kStage;
    constexpr bool kCompact = sizeof(E) == 2;
    static_assert(kWXW == 16, "the query slot layout holds 16 words");
    static_assert(kSec <= 16, "carry counts take 4 bits of the slot");
    __shared__ WarpRows s_rows[kXPB];
    __shared__ __align__(16) uint32_t s_slot[kXPB][32 * kXS];
    __shared__ __align__(16) E s_stage[kXPB][2][kStage];
    __shared__ E s_carry[kXPB][kWQ][kSec];
    E* const nbr = reinterpret_cast<E*>(a.nbr);

    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const uint32_t lsh = 31u - (uint32_t)lane;
    WarpRows& rows = s_rows[wib];
    uint32_t* slots = s_slot[wib];
    const EpsParams* __restrict__ ep = a.ep;
    const int rho = ep->rho;
    const int nrows = 2 * rho + 1;
    const float wf = a.ep->wf;
    const uint32_t nunits = min(*a.nunits, a.unit_hi);  // up to the row chunk's last
    if (a.n <= kSmallFused)
        for (uint64_t k = a.row_lo + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < a.row_hi;
             k += (uint64_t)gridDim.x * blockDim.x)
            small_expand<E>(a, (uint32_t)k);
    __syncwarp();
    const uint32_t ncx_pad = a.g.ncx_pad, G = a.g.G;
    uint32_t par = 0;        // staging buffer of the next query
    uint32_t pending = 0;    // bit b: a copy from buffer b may still be reading it
    uint32_t last_copy = 0;  // buffer of the most recent copy
    const uint32_t stage_s = (uint32_t)__cvta_generic_to_shared(&s_stage[wib][0][0]);

    for (;;) {
        uint32_t u = 0;
        if (lane == 0) u = a.unit_lo + atomicAdd(a.tile_counter, 1u);
        u = __shfl_sync(kFull, u, 0);
        if (u >= nunits) break;
        const uint32_t t = a.ulist[u];
        const uint32_t u0 = a.tile_uoff[t];
        const uint32_t qs = a.tiles[t], qe = a.tiles[t + 1];
        if (!(qs < qe && qe <= a.n && qe - qs <= kUnitQ && u0 <= u)) {
            if (lane == 0) guard_fail(a.st, 4, ((unsigned long long)qs << 32) | qe);
            continue;
        }
        const uint32_t Q = qe - qs;
        const uint32_t key0 = a.gkey[qs];
        const uint32_t cy = key0 / ncx_pad;
        const uint32_t cx0 = (key0 - cy * ncx_pad) / G * G;
        warp_rows(a, ep, rho, nrows, cy, cx0, wf, rows, lane, t);
        const uint32_t C = rows.off[nrows];
        const uint32_t words = (C + 31u) >> 5;
        const uint32_t wbeg = (u - u0) * a.unit_words;
        const uint32_t wend = min(words, wbeg + a.unit_words);
        const unsigned long long bm0 = a.tile_boff[t];
        // row cursors: lane l holds queries l and l+32
        const bool v0 = qs + lane < qe, v1 = qs + lane + 32 < qe;
        unsigned long long cur0 = v0 ? a.off[qs + lane] - a.off_base : 0;
        unsigned long long cur1 = v1 ? a.off[qs + lane + 32] - a.off_base : 0;
        for (uint32_t uu = u0; uu < u; uu++) {
            if (v0) cur0 += a.parts[(unsigned long long)uu * kUnitQ + lane];
            if (v1) cur1 += a.parts[(unsigned long long)uu * kUnitQ + lane + 32];
        }
        // entries staged but not yet written (carried to the next round)
        uint32_t nc0 = 0, nc1 = 0;
        for (uint32_t w0 = wbeg; w0 < wend; w0 += kWXW) {
            const uint32_t nw = min((uint32_t)kWXW, wend - w0);
            const bool last = w0 + kWXW >= wend;  // the unit's last round: write everything
            // entry of each lane's candidate of the round's words: its
            // cell-ordered index, or (compact) its position in the unit
            E id[kWXW];
#pragma unroll
            for (int s = 0; s < kWXW; s++) {
                const uint32_t g = (w0 + (uint32_t)s) * 32u + (uint32_t)lane;
                id[s] = 0;
                if (g < C) {
                    if (kCompact) {
                        id[s] = (E)((w0 - wbeg + (uint32_t)s) * 32u + (uint32_t)lane);
                    } else {
                        int i;
                        id[s] = (E)tile_candidate(rows.start, rows.off, nrows, g, &i);
                    }
                }
            }
            const uint32_t* bw = a.bitmap + bm0 + (unsigned long long)w0 * Q;
            for (uint32_t qh = 0; qh < Q; qh += 32) {
                const uint32_t q = qh + (uint32_t)lane;
                __syncwarp();  // the previous slots have been read
                const bool wrow = qh == 0 ? v0 : v1;
                uint32_t todo = __ballot_sync(kFull, wrow);  // queries whose rows are written
                if (wrow) {
                    uint32_t wd[kWXW], pm[kWXW];
#pragma unroll
                    for (int s = 0; s < kWXW; s++)
                        wd[s] = ((uint32_t)s < nw) ? __ldg(bw + (unsigned long long)s * Q + q) : 0u;
                    const unsigned long long cur = qh == 0 ? cur0 : cur1;
                    const uint32_t nc = qh == 0 ? nc0 : nc1;
                    // table entry wcur + k sits at staging position
                    // (wcur mod kVec) + k: the carried entries first, then this round's
                    const unsigned long long wcur = cur - nc;
                    uint32_t acc = ((uint32_t)wcur & (kVec - 1u)) + nc;
                    // the staging buffer of this query (queries take the two
                    // buffers in turn, in increasing order); pm[s] = shared
                    // address of the entry before word s's first
                    const uint32_t bq = par ^ (__popc(todo & ((1u << lane) - 1u)) & 1u);
                    const uint32_t sbase = stage_s + bq * (uint32_t)(kStage * sizeof(E));
#pragma unroll
                    for (int s = 0; s < kWXW; s++) {
                        pm[s] = sbase + (uint32_t)sizeof(E) * (acc - 1u);
                        acc += __popc(wd[s]);
                    }
                    const uint32_t nstage = acc - ((uint32_t)wcur & (kVec - 1u));  // carried + new
                    const unsigned long long end = wcur + nstage;
                    // written this round: up to the last 32-byte boundary (all at
                    // the unit's last round), never before wcur
                    unsigned long long wto = last ? end : (end & ~(unsigned long long)(kSec - 1u));
                    if (wto < wcur) wto = wcur;
                    const uint32_t nwrite = (uint32_t)(wto - wcur);
                    uint4* sl = reinterpret_cast<uint4*>(slots + lane * kXS);
#pragma unroll
                    for (int v = 0; v < 4; v++) {
                        sl[v] = make_uint4(wd[4 * v], wd[4 * v + 1], wd[4 * v + 2], wd[4 * v + 3]);
                        sl[4 + v] = make_uint4(pm[4 * v], pm[4 * v + 1], pm[4 * v + 2], pm[4 * v + 3]);
                    }
                    sl[8] = make_uint4((uint32_t)wcur, (uint32_t)(wcur >> 32), nstage, nc | (nwrite << 4));
                    if (qh == 0) {
                        cur0 = end;
                        nc0 = nstage - nwrite;
                    } else {
                        cur1 = end;
                        nc1 = nstage - nwrite;
                    }
                }
                __syncwarp();
                for (; todo; todo &= todo - 1u) {
                    const uint32_t qi = (uint32_t)__ffs(todo) - 1u;
                    const uint4* sl = reinterpret_cast<const uint4*>(slots + qi * kXS);
                    uint32_t W[kWXW], P[kWXW];
#pragma unroll
                    for (int v = 0; v < 4; v++) {
                        const uint4 w4 = sl[v], p4 = sl[4 + v];
                        W[4 * v] = w4.x; W[4 * v + 1] = w4.y; W[4 * v + 2] = w4.z; W[4 * v + 3] = w4.w;
                        P[4 * v] = p4.x; P[4 * v + 1] = p4.y; P[4 * v + 2] = p4.z; P[4 * v + 3] = p4.w;
                    }
                    const uint4 cc = sl[8];
                    const unsigned long long wcur = ((unsigned long long)cc.y << 32) | cc.x;
                    const uint32_t nstage = cc.z, nc = cc.w & 15u, nwrite = cc.w >> 4;
                    E* const carry = s_carry[wib][qh + qi];
                    // a copy from this buffer must have read it: if it is the
                    // latest copy, wait for all copies, else for all but one
                    const uint32_t b = par;
                    E* const buf = s_stage[wib][b];
                    par ^= 1u;
                    if (pending & (1u << b)) {
                        if (lane == 0) {
                            if (last_copy == b)
                                asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                            else
                                asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                        }
                        pending &= ~(1u << b);
                    }
                    __syncwarp();
                    // table entry wcur + k sits at buf[phase + k]
                    const uint32_t phase = (uint32_t)wcur & (kVec - 1u);
                    if ((uint32_t)lane < nc) buf[phase + lane] = carry[lane];
#pragma unroll
                    for (int wi = 0; wi < kWXW; wi++) {
                        const uint32_t x = W[wi] << lsh;
                        st_shared_if_neg((int)x, P[wi] + (uint32_t)sizeof(E) * __popc(x), id[wi]);
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    const unsigned long long wto = wcur + nwrite;
                    const unsigned long long A = (wcur + (kVec - 1u)) & ~(unsigned long long)(kVec - 1u);
                    const unsigned long long B = wto & ~(unsigned long long)(kVec - 1u);
                    E* const sb = buf + phase;
                    if (B > A) {
                        if (lane == 0)
                            bulk_copy_to_global(nbr + A, sb + (uint32_t)(A - wcur),
                                                (uint32_t)(B - A) * (uint32_t)sizeof(E));
                        pending |= 1u << b;
                        last_copy = b;
                        const uint32_t nh = (uint32_t)(A - wcur), nt = (uint32_t)(wto - B);
                        if ((uint32_t)lane < nh)
                            nbr[wcur + (uint32_t)lane] = sb[lane];
                        else if ((uint32_t)lane >= kVec && (uint32_t)lane - kVec < nt)
                            nbr[B + ((uint32_t)lane - kVec)] = sb[(uint32_t)(B - wcur) + ((uint32_t)lane - kVec)];
                    } else if ((uint32_t)lane < nwrite) {
                        nbr[wcur + (uint32_t)lane] = sb[lane];  // fewer than 2 kVec - 1 entries
                    }
                    // entries after the last 32-byte boundary wait for the next round
                    if ((uint32_t)lane < nstage - nwrite) carry[lane] = sb[nwrite + (uint32_t)lane];
                }
            }
        }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// The words of a block of 32 (the first is word w0 of the tile's, of C
// candidates) that a 16-bit table's rows get as runs: full words (inside, as
// the count pass flagged them) in a row of three or more.  Shorter runs cost
// less among the words that are expanded; the tile's last word, if it has
// fewer than 32 candidates, is no full one.  Within a unit, a row holds the
// other words' entries first, in order, then the runs'.
__device__ __forceinline__ uint32_t full_runs(uint32_t inside, uint32_t w0, uint32_t C) {
    const uint32_t whole = (C >> 5) > w0 ? (C >> 5) - w0 : 0u;  // words of 32 candidates
    const uint32_t F = whole >= 32u ? inside : inside & ((1u << whole) - 1u);
    const uint32_t starts = F & (F >> 1) & (F >> 2);
    return starts | (starts << 1) | (starts << 2);
}

// A run of full words of a 16-bit table (len candidates, up to 16 words): all
// are neighbours of every query, their boxes lie inside eps of the whole tile.
// All rows get the same run of ids, at their own places: lane = query writes the entries
// carried from its last round and those up to the next 16-byte boundary, and
// copies the rest straight from one of eight staged runs, the one that starts
// with the id that falls on the boundary.  Four runs at a time fit the slots'
// memory.  cur: the row's place of id0, nc entries are carried before it; the
// row is written up to its last 32-byte boundary (last: up to its end) and the
// entries after that are carried.  A run is 3 words or more, but cut into pieces
// of 16: len is at least 32.
__device__ __noinline__ void full_round(uint16_t* __restrict__ nbr, uint32_t* slots,
                                        uint16_t* carry, bool wrow, uint32_t id0, uint32_t len, bool last,
                                        unsigned long long cur, uint32_t nc, int lane) {
    constexpr uint32_t kRun = kWXW * 32u;
    static_assert(4u * kRun * sizeof(uint16_t) <= 32u * kXS * sizeof(uint32_t), "four runs fit");
    const unsigned long long wcur = cur - nc, end = cur + len;
    const unsigned long long A = (cur + 7ull) & ~7ull;
    const unsigned long long wto = last ? end : end & ~15ull;  // (past A: len >= 32)
    const unsigned long long B = wto & ~7ull;
    const uint32_t first = (uint32_t)(A - cur);  // entries of the run before A
    if (wrow) {
        const uint32_t n0 = (uint32_t)(A - wcur);
        auto entry = [&](uint32_t i) {
            return i < nc ? (uint32_t)carry[i] : id0 + (i - nc);
        };
        if (((uint32_t)wcur & 7u) == 0u) {
            for (uint32_t i = 0; i < n0; i += 8) {
                uint4 v;
                v.x = entry(i) | (entry(i + 1) << 16);
                v.y = entry(i + 2) | (entry(i + 3) << 16);
                v.z = entry(i + 4) | (entry(i + 5) << 16);
                v.w = entry(i + 6) | (entry(i + 7) << 16);
                *reinterpret_cast<uint4*>(nbr + wcur + i) = v;
            }
        } else {
            for (uint32_t i = 0; i < n0; i++) nbr[wcur + i] = (uint16_t)entry(i);
        }
        for (unsigned long long i = B; i < wto; i++) nbr[i] = (uint16_t)(id0 + (uint32_t)(i - cur));
        for (unsigned long long i = wto; i < end; i++)
            carry[i - wto] = (uint16_t)(id0 + (uint32_t)(i - cur));
    }
#pragma unroll 1
    for (uint32_t b = 0; b < 2; b++) {
        const bool mine = wrow && (first >> 2) == b;
        if (!__any_sync(kFull, mine)) continue;
        if (b) {  // the first four runs have been read
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            __syncwarp();
        }
        for (uint32_t v = (uint32_t)lane; v < kRun / 2; v += 32) {
            const uint32_t run = v / (kRun / 8), at = v % (kRun / 8);
            const uint32_t x = id0 + 4u * b + run + 8u * at;
            const uint32_t two = x * 0x10001u + 0x10000u;  // x, x + 1
            reinterpret_cast<uint4*>(slots)[run * (kRun / 8) + at] =
                make_uint4(two, two + 0x20002u, two + 0x40004u, two + 0x60006u);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (mine && B > A)
            bulk_copy_to_global(nbr + A, slots + (first & 3u) * (kRun / 2),
                                (uint32_t)(B - A) * (uint32_t)sizeof(uint16_t));
    }
}

// 16-bit tables.  The count pass flags the words that are outside eps of the
// whole tile (skipped here) and those inside it (runs of three or more are
// copied from staged runs of ids, full_round); the others are packed into
// rounds of 16 words.  Two queries per pass: the round's words are transposed
// into the query slots as above (lane = query); then lanes 0-15 expand one
// query of a pair and lanes 16-31 the other, lane j of a half taking bits j
// and j + 16 of every word.  The work of a query that does not depend on its
// words (slot reads, barriers, the proxy fence, the bulk copy, the head and
// tail stores, the carry) is thus done once per two queries.  One staging
// buffer per half: before a half stages its next query, its first lane waits
// until its copies have read the buffer (bulk async-groups belong to the
// issuing thread).  With one buffer per half and no per-warp row table (the
// 16-bit entries need only the tile's candidate count), 8 blocks of 3 warps
// (80 registers, 26.4 KB of shared memory) share an SM; the extra warps hide
// more of the kernel's dependency latency (2M sweep: 34.7 ms of tables against
// 40.3 with two buffers per half at 6 blocks).  Bound by the issue of shared
// stores where most words are mixed, by the table's writes where most are
// whole: 1M sweep, eps 0.1 / 0.2 / 0.4 / 0.8: 0.26 / 0.53 / 1.10 / 2.67 ms, 1.0
// to 4.7 TB/s of entries (eps 0.8 3.24 ms before the runs were copied).
__global__ void __launch_bounds__(kXPB * 32, 8) expand16_kernel(TableArgs a) {
    pdl_sync();
    using E = uint16_t;
    constexpr uint32_t kVec = XFmt<E>::kVec, kSec = XFmt<E>::kSec, kStage = XFmt<E>::kStage;
    static_assert(kWXW == 16, "the query slot layout holds 16 words");
    static_assert(kSec <= 16 && 2 * kVec <= 16, "head, tail and carry fit a half-warp");
    __shared__ __align__(16) uint32_t s_slot[kXPB][32 * kXS];
    __shared__ __align__(16) E s_stage[kXPB][2][kStage];
    __shared__ E s_carry[kXPB][kWQ][kSec];
    __shared__ __align__(16) uint8_t s_list[kXPB][kUnitWords];
    E* const nbr = reinterpret_cast<E*>(a.nbr);

    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const uint32_t hj = (uint32_t)lane & 15u, half = (uint32_t)lane >> 4;
    const uint32_t lsh_a = 31u - hj, lsh_b = 15u - hj;  // bit hj, bit hj + 16 to the sign
    uint32_t* slots = s_slot[wib];
    const EpsParams* __restrict__ ep = a.ep;
    const int rho = ep->rho;
    const int nrows = 2 * rho + 1;
    const uint32_t nunits = min(*a.nunits, a.unit_hi);
    if (a.n <= kSmallFused)
        for (uint64_t k = a.row_lo + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < a.row_hi;
             k += (uint64_t)gridDim.x * blockDim.x)
            small_expand<E>(a, (uint32_t)k);
    __syncwarp();
    const uint32_t ncx_pad = a.g.ncx_pad, G = a.g.G;
    uint32_t pending = 0;    // nonzero: a copy from this half's buffer may be reading it
    uint32_t slot_copies = 0;  // nonzero: copies of a full round may be reading the slots
    const uint32_t stage_s = (uint32_t)__cvta_generic_to_shared(&s_stage[wib][0][0]);

    for (;;) {
        uint32_t u = 0;
        if (lane == 0) u = a.unit_lo + atomicAdd(a.tile_counter, 1u);
        u = __shfl_sync(kFull, u, 0);
        if (u >= nunits) break;
        const uint32_t t = a.ulist[u];
        const uint32_t u0 = a.tile_uoff[t];
        const uint32_t qs = a.tiles[t], qe = a.tiles[t + 1];
        if (!(qs < qe && qe <= a.n && qe - qs <= kUnitQ && u0 <= u)) {
            if (lane == 0) guard_fail(a.st, 4, ((unsigned long long)qs << 32) | qe);
            continue;
        }
        const uint32_t Q = qe - qs;
        const uint32_t key0 = a.gkey[qs];
        const uint32_t cy = key0 / ncx_pad;
        const uint32_t cx0 = (key0 - cy * ncx_pad) / G * G;
        // candidates of the tile (16-bit entries are positions: the rows'
        // starts are not needed here)
        uint32_t Cl = 0;
        for (int i = lane; i < nrows; i += 32) {
            uint32_t st, len, base;
            tile_row(a, ep, rho, cy, cx0, i, &st, &len, &base, t);
            Cl += len;
        }
        const uint32_t C = __reduce_add_sync(kFull, Cl);
        const uint32_t words = (C + 31u) >> 5;
        const uint32_t wbeg = (u - u0) * a.unit_words;
        const uint32_t wend = min(words, wbeg + a.unit_words);
        const unsigned long long bm0 = a.tile_boff[t];
        const bool v0 = qs + lane < qe, v1 = qs + lane + 32 < qe;
        unsigned long long cur0 = v0 ? a.off[qs + lane] - a.off_base : 0;
        unsigned long long cur1 = v1 ? a.off[qs + lane + 32] - a.off_base : 0;
        for (uint32_t uu = u0; uu < u; uu++) {
            if (v0) cur0 += a.parts[(unsigned long long)uu * kUnitQ + lane];
            if (v1) cur1 += a.parts[(unsigned long long)uu * kUnitQ + lane + 32];
        }
        // The unit's words in blocks of 32 (lane b: block b): first those to
        // expand, then the runs of full words.
        uint32_t mix = 0u, run = 0u;
        if ((uint32_t)lane * 32u < wend - wbeg) {
            const uint32_t w0 = wbeg + 32u * (uint32_t)lane;
            const uint2 f = a.wflags[(unsigned long long)u * flag_blocks(a.unit_words) + lane];
            const uint32_t nwb = min(32u, wend - w0);
            run = full_runs(f.x, w0, C);
            mix = (nwb == 32u ? kFull : (1u << nwb) - 1u) & ~f.y & ~run;
        }
        uint8_t* const list = s_list[wib];
        uint32_t nmix = 0;
        __syncwarp();  // (the list before has been read)
#pragma unroll
        for (uint32_t b = 0; b < kUnitWords / 32u; b++) {
            const uint32_t m = __shfl_sync(kFull, mix, (int)b);
            if ((m >> lane) & 1u)
                list[nmix + __popc(m & ((1u << lane) - 1u))] = (uint8_t)(32u * b + (uint32_t)lane);
            nmix += (uint32_t)__popc(m);
        }
        __syncwarp();
        const uint32_t run_blocks = __ballot_sync(kFull, run != 0u);
        const uint32_t* bw = a.bitmap + bm0 + (unsigned long long)wbeg * Q;
        for (uint32_t qh = 0; qh < Q; qh += 32) {
            const uint32_t q = qh + (uint32_t)lane;
            const bool wrow = qh == 0 ? v0 : v1;
            unsigned long long cur = qh == 0 ? cur0 : cur1;
            uint32_t nc = 0;
            for (uint32_t r0 = 0; r0 < nmix; r0 += kWXW) {
                uint32_t todo = __ballot_sync(kFull, wrow);
                const uint32_t nw = min((uint32_t)kWXW, nmix - r0);
                const bool last = r0 + kWXW >= nmix && run_blocks == 0u;
                if (slot_copies) {
                    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                    pending = 0;
                    slot_copies = 0;
                }
                __syncwarp();  // the previous slots have been read
                // the round's words, and the ids of bit hj of words 2i (low
                // half) and 2i + 1 (bit hj + 16: + 16): positions in the unit
                uint32_t l4[4];
                {
                    const uint4 v = *reinterpret_cast<const uint4*>(list + r0);
                    l4[0] = v.x; l4[1] = v.y; l4[2] = v.z; l4[3] = v.w;
                }
                uint32_t ids2[kWXW / 2];
#pragma unroll
                for (int i = 0; i < kWXW / 2; i++) {
                    const uint32_t pair = l4[i >> 1] >> (16 * (i & 1));
                    ids2[i] = ((pair & 127u) * 32u + hj) | ((((pair >> 8) & 127u) * 32u + hj) << 16);
                }
                if (wrow) {
                    uint32_t wd[kWXW], pm[kWXW];
#pragma unroll
                    for (int s = 0; s < kWXW; s++) {
                        const uint32_t at = (l4[s >> 2] >> (8 * (s & 3))) & 127u;
                        wd[s] = (uint32_t)s < nw ? __ldg(bw + (unsigned long long)at * Q + q) : 0u;
                    }
                    const unsigned long long wcur = cur - nc;
                    uint32_t acc = ((uint32_t)wcur & (kVec - 1u)) + nc;
                    // the k-th query of todo is expanded in pass k / 2 by half
                    // k % 2, in that half's buffer
                    const uint32_t k = __popc(todo & ((1u << lane) - 1u));
                    const uint32_t bq = k & 1u;
                    const uint32_t sbase = stage_s + bq * (uint32_t)(kStage * sizeof(E));
#pragma unroll
                    for (int s = 0; s < kWXW; s++) {
                        pm[s] = sbase + (uint32_t)sizeof(E) * (acc - 1u);
                        acc += __popc(wd[s]);
                    }
                    const uint32_t nstage = acc - ((uint32_t)wcur & (kVec - 1u));
                    const unsigned long long end = wcur + nstage;
                    unsigned long long wto = last ? end : (end & ~(unsigned long long)(kSec - 1u));
                    if (wto < wcur) wto = wcur;
                    const uint32_t nwrite = (uint32_t)(wto - wcur);
                    uint4* sl = reinterpret_cast<uint4*>(slots + lane * kXS);
#pragma unroll
                    for (int v = 0; v < 4; v++) {
                        sl[v] = make_uint4(wd[4 * v], wd[4 * v + 1], wd[4 * v + 2], wd[4 * v + 3]);
                        sl[4 + v] = make_uint4(pm[4 * v], pm[4 * v + 1], pm[4 * v + 2], pm[4 * v + 3]);
                    }
                    sl[8] = make_uint4((uint32_t)wcur, (uint32_t)(wcur >> 32), nstage, nc | (nwrite << 4));
                    cur = end;
                    nc = nstage - nwrite;
                }
                __syncwarp();
                while (todo) {
                    const uint32_t qa = (uint32_t)__ffs(todo) - 1u;
                    todo &= todo - 1u;
                    const bool has_b = todo != 0u;
                    const uint32_t qb = has_b ? (uint32_t)__ffs(todo) - 1u : qa;
                    if (has_b) todo &= todo - 1u;
                    const bool act = half == 0u || has_b;  // the second half idles on an odd count
                    const uint32_t qi = half ? qb : qa;
                    const uint4* sl = reinterpret_cast<const uint4*>(slots + qi * kXS);
                    uint32_t W[kWXW], P[kWXW];
#pragma unroll
                    for (int v = 0; v < 4; v++) {
                        const uint4 w4 = sl[v], p4 = sl[4 + v];
                        W[4 * v] = w4.x; W[4 * v + 1] = w4.y; W[4 * v + 2] = w4.z; W[4 * v + 3] = w4.w;
                        P[4 * v] = p4.x; P[4 * v + 1] = p4.y; P[4 * v + 2] = p4.z; P[4 * v + 3] = p4.w;
                    }
                    const uint4 cc = sl[8];
                    const unsigned long long wcur = ((unsigned long long)cc.y << 32) | cc.x;
                    const uint32_t nstage = cc.z, nc = cc.w & 15u, nwrite = cc.w >> 4;
                    E* const carry = s_carry[wib][qh + qi];
                    E* const buf = s_stage[wib][half];
                    // the half's copies must have read its buffer
                    if (act && pending) {
                        if (hj == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                        pending = 0;
                    }
                    __syncwarp();
                    const uint32_t phase = (uint32_t)wcur & (kVec - 1u);
                    if (act) {
                        if (hj < nc) buf[phase + hj] = carry[hj];
#pragma unroll
                        for (int wi = 0; wi < kWXW; wi++) {
                            const uint32_t xa = W[wi] << lsh_a, xb = W[wi] << lsh_b;
                            const uint32_t id = (wi & 1) ? ids2[wi >> 1] >> 16 : ids2[wi >> 1];
                            st_shared_if_neg((int)xa, P[wi] + (uint32_t)sizeof(E) * __popc(xa), (E)id);
                            st_shared_if_neg((int)xb, P[wi] + (uint32_t)sizeof(E) * __popc(xb),
                                             (E)(id + 16u));
                        }
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (act) {
                        const unsigned long long wto = wcur + nwrite;
                        const unsigned long long A = (wcur + (kVec - 1u)) & ~(unsigned long long)(kVec - 1u);
                        const unsigned long long B = wto & ~(unsigned long long)(kVec - 1u);
                        E* const sb = buf + phase;
                        if (B > A) {
                            if (hj == 0)
                                bulk_copy_to_global(nbr + A, sb + (uint32_t)(A - wcur),
                                                    (uint32_t)(B - A) * (uint32_t)sizeof(E));
                            pending = 1u;
                            const uint32_t nh = (uint32_t)(A - wcur), nt = (uint32_t)(wto - B);
                            if (hj < nh)
                                nbr[wcur + hj] = sb[hj];
                            else if (hj >= kVec && hj - kVec < nt)
                                nbr[B + (hj - kVec)] = sb[(uint32_t)(B - wcur) + (hj - kVec)];
                        } else if (hj < nwrite) {
                            nbr[wcur + hj] = sb[hj];  // fewer than 2 kVec - 1 entries
                        }
                        if (hj < nstage - nwrite) carry[hj] = sb[nwrite + hj];
                    }
                }
            }
            __syncwarp();  // (the carries have been written)
            for (uint32_t bl = run_blocks; bl; bl &= bl - 1u) {
                const uint32_t b = (uint32_t)__ffs(bl) - 1u;
                for (uint32_t rem = __shfl_sync(kFull, run, (int)b); rem;) {
                    const uint32_t w = (uint32_t)__ffs(rem) - 1u;
                    // (32 words of a run: ffs(0) - 1 is larger than any)
                    const uint32_t k = min((uint32_t)__ffs(~(rem >> w)) - 1u, (uint32_t)kWXW);
                    rem &= ~(((1u << k) - 1u) << w);
                    if (slot_copies) {
                        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                        pending = 0;
                    }
                    __syncwarp();
                    const bool last = rem == 0u && (bl & (bl - 1u)) == 0u;
                    full_round(nbr, slots, s_carry[wib][qh + lane], wrow, (32u * b + w) * 32u, 32u * k,
                               last, cur, nc, lane);
                    slot_copies = 1;
                    cur += 32u * k;
                    nc = last ? 0u : (uint32_t)cur & (kSec - 1u);
                }
            }
        }
    }
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// Table pass without a bitmap: a block per tile re-tests its candidates and
// writes each query's row (off, off_base).  The tests are the count pass's, the
// FP32 ones on the plain squared distance.
template <bool MIXED>
__global__ void __launch_bounds__(kTT) fill_kernel(TableArgs a) {
    pdl_sync();
    __shared__ float2 s_rel[kChunk];
    __shared__ double2 s_xy[kChunk];
    __shared__ uint32_t s_id[kChunk];
    __shared__ uint32_t s_seg_start[kMaxRows];
    __shared__ uint32_t s_seg_off[kMaxRows + 1];
    __shared__ uint32_t s_seg_base[kMaxRows];
    __shared__ float s_seg_dyw[kMaxRows];
    __shared__ uint32_t s_tile;

    const int tid = threadIdx.x, lane = tid & 31;
    const uint32_t lt = (1u << lane) - 1u;
    const EpsParams* __restrict__ ep = a.ep;
    const double thr = ep->thr, tbox = ep->tbox;
    const ExactBounds xb = ep->xb;
    const float lo = ep->lo32, hi = ep->hi32;
    const int rho = ep->rho;
    const int nrows = 2 * rho + 1;
    const float wf = a.ep->wf;
    const uint32_t tile_end = a.tile_end != 0xffffffffu ? a.tile_end : *a.ntiles;
    const uint32_t ncx_pad = a.g.ncx_pad, G = a.g.G;
    unsigned long long my_retest = 0;

    for (;;) {
        if (tid == 0) s_tile = a.tile_lo + atomicAdd(a.tile_counter, 1u);
        __syncthreads();
        const uint32_t t = s_tile;
        if (t >= tile_end) break;
        const uint32_t qs = a.tiles[t], qe = a.tiles[t + 1];
        if (!(qs < qe && qe <= a.n)) {
            if (tid == 0) guard_fail(a.st, 1, ((unsigned long long)qs << 32) | qe);
            __syncthreads();
            continue;
        }
        const uint32_t key0 = a.gkey[qs];
        const uint32_t cy = key0 / ncx_pad;
        const uint32_t cx0 = (key0 - cy * ncx_pad) / G * G;
        const uint32_t tile_base = cy * ncx_pad + cx0;

        if (tid < nrows) {
            uint32_t st, len, base;
            tile_row(a, ep, rho, cy, cx0, tid, &st, &len, &base);
            s_seg_start[tid] = st;
            s_seg_off[tid + 1] = len;
            s_seg_base[tid] = base;
            s_seg_dyw[tid] = __fmul_rn((float)(tid - rho), wf);
        }
        __syncthreads();
        if (tid == 0) {
            uint32_t acc = 0;
            s_seg_off[0] = 0;
            for (int i = 0; i < nrows; i++) {
                acc += s_seg_off[i + 1];
                s_seg_off[i + 1] = acc;
            }
        }
        __syncthreads();
        const uint32_t C = s_seg_off[nrows];

        // queries of this thread: lane l of warp w takes tile queries 64 w + l and
        // 64 w + 32 + l, so a small tile fills the slots of its first warps, the
        // other warps skip the tests, and a tile of up to 32 queries tests one a
        // lane (two on half of the lanes took as long as 64 queries do: 50k
        // points in one cell, 16-bit table without a bitmap, 127 -> 104 ms)
        const uint32_t q0 = qs + (uint32_t)(tid & ~31) * kQPT + (uint32_t)lane;
        const bool warp_active = qs + (uint32_t)(tid & ~31) * kQPT < qe;
        const bool two = qs + (uint32_t)(tid & ~31) * kQPT + 32u < qe;
        float qx[kQPT], qy[kQPT];
        double2 qd[kQPT];
        uint32_t qk[kQPT];
        unsigned long long cur[kQPT], rend[kQPT];
#pragma unroll
        for (int q = 0; q < kQPT; q++) {
            const uint32_t k = q0 + 32u * q;
            qk[q] = k;
            cur[q] = rend[q] = 0;
            if (k < qe) {
                const float2 loc = a.glocal[k];
                const int dcx = (int)(a.gkey[k] - tile_base);
                qx[q] = __fmaf_rn((float)dcx, wf, loc.x);
                qy[q] = loc.y;
                qd[q] = a.gxy[k];
                cur[q] = a.off[k] - a.off_base;
                rend[q] = a.off[k + 1] - a.off_base;
            } else {
                qx[q] = qy[q] = __int_as_float(0x7fc00000);
                qd[q] = make_double2(__longlong_as_double(0x7ff8000000000000ll),
                                     __longlong_as_double(0x7ff8000000000000ll));
            }
        }

        for (uint32_t cb = 0; cb < C; cb += kChunk) {
            const uint32_t len = min((uint32_t)kChunk, C - cb);
            const uint32_t len32 = (len + 31u) & ~31u;
            for (uint32_t j = tid; j < len32; j += kTT) {
                uint32_t k = 0xffffffffu;
                int i = 0;
                if (j < len) {
                    k = tile_candidate(s_seg_start, s_seg_off, nrows, cb + j, &i);
                    if (!VDB_GUARD(a.st, k < a.n, 3, k)) k = 0xffffffffu;
                }
                if (k != 0xffffffffu) {
                    if (MIXED) {
                        const float2 loc = a.glocal[k];
                        const int dcx = (int)(a.gkey[k] - s_seg_base[i]);
                        s_rel[j] = make_float2(__fmaf_rn((float)dcx, wf, loc.x),
                                               __fadd_rn(loc.y, s_seg_dyw[i]));
                    }
                    s_xy[j] = a.gxy[k];
                    s_id[j] = k;
                } else {
                    // padding: NaN fails every comparison (also against thr = inf)
                    s_rel[j] = make_float2(__int_as_float(0x7fc00000), __int_as_float(0x7fc00000));
                    s_xy[j] = make_double2(__longlong_as_double(0x7ff8000000000000ll),
                                           __longlong_as_double(0x7ff8000000000000ll));
                    s_id[j] = 0;
                }
            }
            __syncthreads();

            for (uint32_t j0 = 0; warp_active && j0 < len; j0 += 32) {
                uint32_t m[kQPT], hm[kQPT];
#pragma unroll
                for (int q = 0; q < kQPT; q++) m[q] = hm[q] = 0u;
#pragma unroll
                for (int jj = 0; jj < 32; jj++) {
                    if (MIXED) {
                        const float2 c = s_rel[j0 + jj];
#pragma unroll
                        for (int q = 0; q < kQPT; q++) {
                            if (q == 1 && !two) break;
                            const float dx = __fsub_rn(qx[q], c.x);
                            const float dy = __fsub_rn(qy[q], c.y);
                            const float d2 = __fmaf_rn(dx, dx, __fmul_rn(dy, dy));
                            m[q] |= (d2 < lo) ? (1u << jj) : 0u;
                            hm[q] |= (d2 <= hi) ? (1u << jj) : 0u;
                        }
                    } else {
                        const double2 c = s_xy[j0 + jj];
#pragma unroll
                        for (int q = 0; q < kQPT; q++) {
                            if (q == 1 && !two) break;
                            const double dx = __dsub_rn(qd[q].x, c.x);
                            const double dy = __dsub_rn(qd[q].y, c.y);
                            const double d2 = __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy));
                            m[q] |= (d2 <= tbox) ? (1u << jj) : 0u;
                            hm[q] |= (d2 <= thr) ? (1u << jj) : 0u;
                        }
                    }
                }
                // pairs in the band: exact FP64 predicate
                uint32_t amb[kQPT], asy[kQPT], any = 0u;
#pragma unroll
                for (int q = 0; q < kQPT; q++) {
                    amb[q] = hm[q] & ~m[q];
                    asy[q] = 0u;
                    any |= amb[q];
                }
                if (__any_sync(kFull, any != 0u)) {
#pragma unroll
                    for (int q = 0; q < kQPT; q++) {
                        while (amb[q]) {
                            const int jj = __ffs(amb[q]) - 1;
                            amb[q] &= amb[q] - 1u;
                            const uint32_t kq = s_id[j0 + jj];
                            const uint32_t r = exact_pair(qd[q], s_xy[j0 + jj], qk[q], kq, xb,
                                                          a.gbox);
                            my_retest++;
                            if (r & 1u) {
                                m[q] |= 1u << jj;
                                if (!(r & 2u)) asy[q] |= 1u << jj;
                            }
                        }
                    }
                }
#pragma unroll
                for (int q = 0; q < kQPT; q++) {
                    uint32_t act = __ballot_sync(kFull, m[q] != 0u);
                    while (act) {
                        const int src = __ffs(act) - 1;
                        act &= act - 1u;
                        const uint32_t mm = __shfl_sync(kFull, m[q], src);
                        const uint32_t am = __shfl_sync(kFull, asy[q], src);
                        const unsigned long long c0 = __shfl_sync(kFull, cur[q], src);
                        const unsigned long long ce = __shfl_sync(kFull, rend[q], src);
                        if ((mm >> lane) & 1u) {
                            const unsigned long long dst = c0 + __popc(mm & lt);
                            if (dst < ce) {
                                const bool one_way = (am >> lane) & 1u;
                                if (a.compact)  // position in its work unit's candidates
                                    reinterpret_cast<uint16_t*>(a.nbr)[dst] =
                                        (uint16_t)(((cb + j0 + (uint32_t)lane) &
                                                    (a.unit_words * 32u - 1u)) |
                                                   (one_way ? kAsymFlag16 : 0u));
                                else
                                    a.nbr[dst] = s_id[j0 + lane] | (one_way ? kAsymFlag : 0u);
                            } else {
                                atomicOr(&a.st->flags, kStatRowOverflow);
                            }
                        }
                        if (lane == src) cur[q] += __popc(mm);
                    }
                }
            }
            __syncthreads();
        }
        __syncthreads();
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) my_retest += __shfl_down_sync(kFull, my_retest, d);
    if (lane == 0 && my_retest) atomicAdd(&a.st->retested, my_retest);
}

// Candidate ranges [st[j], en[j]) of kRowBatch rows i0 + j of a tile at cells
// cy, cx0 .. cx0 + G - 1.  The rows' loads, and in sparse grids the steps of
// their searches, are side by side: one after the other they were most of the
// tile-words pass.
constexpr int kRowBatch = 5;
__device__ __forceinline__ void tile_rows(const TableArgs& a, const EpsParams* __restrict__ ep,
                                          int rho, int nrows, uint32_t cy, uint32_t cx0, int i0,
                                          uint32_t (&st)[kRowBatch], uint32_t (&en)[kRowBatch]) {
    uint32_t lo[kRowBatch], hi[kRowBatch];  // columns [lo, hi]
    bool on[kRowBatch];
#pragma unroll
    for (int j = 0; j < kRowBatch; j++) {
        const int i = i0 + j, ry = (int)cy + i - rho;
        on[j] = i < nrows && ry >= 0 && ry < (int)a.g.ncy;
        const int reach = on[j] ? ep->reach[i] : 0;
        lo[j] = (uint32_t)max((int)cx0 - reach, 0);
        hi[j] = (uint32_t)min((int)(cx0 + a.g.G - 1) + reach, (int)a.g.ncx - 1);
        st[j] = en[j] = 0;
    }
    if (!a.g.sparse) {
#pragma unroll
        for (int j = 0; j < kRowBatch; j++) {
            if (!on[j]) continue;
            const uint32_t base = (uint32_t)((int)cy + i0 + j - rho) * a.g.ncx_pad;
            st[j] = a.cell_start[base + lo[j]];
            en[j] = a.cell_start[base + hi[j] + 1];
        }
    } else {
        uint32_t b[kRowBatch], len[kRowBatch], re[kRowBatch];
        bool left = false;
#pragma unroll
        for (int j = 0; j < kRowBatch; j++) {
            const uint32_t ry = on[j] ? (uint32_t)((int)cy + i0 + j - rho) : 0u;
            b[j] = a.crow[ry];
            re[j] = a.crow[ry + 1];
            len[j] = on[j] ? re[j] - b[j] : 0u;
            left |= len[j] != 0u;
        }
        while (left) {
            left = false;
#pragma unroll
            for (int j = 0; j < kRowBatch; j++) {
                const uint32_t half = len[j] >> 1;
                if (len[j]) {
                    if (a.ccx[b[j] + half] < lo[j]) {
                        b[j] += half + 1;
                        len[j] -= half + 1;
                    } else {
                        len[j] = half;
                    }
                }
                left |= len[j] != 0u;
            }
        }
#pragma unroll
        for (int j = 0; j < kRowBatch; j++) {
            if (!on[j]) continue;
            uint32_t e = b[j];
            if (hi[j] - lo[j] <= 16u)
                while (e < re[j] && a.ccx[e] <= hi[j]) e++;
            else
                e = cx_lower_bound(a.ccx, e, re[j], hi[j] + 1);
            st[j] = a.clist[b[j]];
            en[j] = a.clist[e];
        }
    }
#pragma unroll
    for (int j = 0; j < kRowBatch; j++) {
        if (!VDB_GUARD(a.st, st[j] <= en[j] && en[j] <= a.n, 2,
                       ((unsigned long long)st[j] << 32) | en[j]))
            st[j] = en[j] = 0;
    }
}

// A thread per tile: its row segments (kept in trow_s/e where set), the words
// of its test bitmap, ceil(C/32) per query, and its work units,
// ceil(ceil(C/32) / unit_words), or none if it is small; the offsets of both by a
// single-pass scan (boff may be null: no bitmap).  Where there are more units than
// 31 bits hold (dense data of 10^7 points and more; their counts would take 500
// GB), kStatTooManyUnits is set and the offsets are not to be used.  Blocks past
// the last tile only clear their part of deg (and the one-way pairs' counter).
__global__ void __launch_bounds__(kLookThreads) tile_words_kernel(
    TableArgs a, unsigned long long* __restrict__ boff, uint32_t* __restrict__ uoff,
    unsigned long long* __restrict__ nwords, uint32_t* __restrict__ nunits, LookState lu,
    LookState lw) {
    pdl_sync();
    const uint32_t tile = lookback_ticket(lu);
    const uint32_t t = tile * kLookThreads + threadIdx.x;
    if (t < a.n) a.deg[t] = 0u;
    if (t == 0) *a.asym_n = 0u;
    const uint32_t ntiles = *a.ntiles;
    if (tile * kLookThreads >= ntiles) return;  // (the whole block)
    const EpsParams* __restrict__ ep = a.ep;
    const int rho = ep->rho, nrows = 2 * rho + 1;
    unsigned long long w = 0;
    uint32_t nu = 0;
    if (t < ntiles) {
        const uint32_t qs = a.tiles[t], qe = a.tiles[t + 1];
        const uint32_t key0 = a.gkey[qs];
        const uint32_t cy = key0 / a.g.ncx_pad;
        const uint32_t cx0 = (key0 - cy * a.g.ncx_pad) / a.g.G * a.g.G;
        uint32_t c = 0;
        for (int i0 = 0; i0 < nrows; i0 += kRowBatch) {
            uint32_t st[kRowBatch], en[kRowBatch];
            tile_rows(a, ep, rho, nrows, cy, cx0, i0, st, en);
#pragma unroll
            for (int j = 0; j < kRowBatch; j++) {
                c += en[j] - st[j];
                if (a.trow_s && i0 + j < nrows) {
                    const unsigned long long k =
                        (unsigned long long)t * (uint32_t)nrows + (uint32_t)(i0 + j);
                    a.trow_s[k] = st[j];
                    a.trow_e[k] = en[j];
                }
            }
        }
        const uint32_t tw = (c + 31u) >> 5;
        w = (unsigned long long)tw * (qe - qs);
        if (c > (a.mixed ? kSmallCand : kSmallCand64) || qe - qs > kSmallQueries)
            nu = (tw + a.unit_words - 1) / a.unit_words;
        if (w > 0xffffffffull) {
            atomicOr(&a.st->flags, kStatBitmapTooLarge);
            w = 0;
        }
    }
    unsigned long long before[2] = {nu, boff ? w : 0ull};
    unsigned long long* const states[2] = {lu.tiles, lw.tiles};
    block_lookbacks<2>(before, tile, states, a.st);
    if (t < ntiles) {
        const uint32_t u0 = (uint32_t)before[0];
        uoff[t] = u0;
        if (boff) boff[t] = before[1];
        if (t == ntiles - 1) {
            if (before[0] + nu > 0x7fffffffull) atomicOr(&a.st->flags, kStatTooManyUnits);
            uoff[ntiles] = u0 + nu;
            *nunits = u0 + nu;
            if (boff) *nwords = before[1] + w;
        }
    }
}

// ulist: the tile of every unit, a thread per tile, long lists by the whole
// warp.  The first blocks make the word boxes (where there are any), which would
// have no use for a launch of their own.
__global__ void __launch_bounds__(kTT) unit_list_kernel(TableArgs a, uint32_t* ulist,
                                                        uint32_t box_blocks) {
    pdl_sync();
    if (blockIdx.x < box_blocks) {
        word_box(a, blockIdx.x * kTT + threadIdx.x);
        return;
    }
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t ntiles = *a.ntiles;
    const uint32_t t = (blockIdx.x - box_blocks) * kTT + threadIdx.x;
    if (t - lane >= ntiles) return;  // (whole warps)
    uint32_t b = 0, e = 0;
    if (t < ntiles) {
        b = a.tile_uoff[t];
        e = a.tile_uoff[t + 1];
    }
    if (e - b <= 8u)
        for (uint32_t i = b; i < e; i++) ulist[i] = t;
    for (uint32_t l = __ballot_sync(kFull, e - b > 8u); l; l &= l - 1u) {
        const int src = __ffs(l) - 1;
        const uint32_t bb = __shfl_sync(kFull, b, src), ee = __shfl_sync(kFull, e, src);
        for (uint32_t i = bb + lane; i < ee; i += 32) ulist[i] = t - lane + (uint32_t)src;
    }
}

// splitmix64 finaliser (a published 64-bit mixer).
__device__ __forceinline__ unsigned long long mix64(unsigned long long x) {
    x ^= x >> 30;
    x *= 0xbf58476d1ce4e5b9ull;
    x ^= x >> 27;
    x *= 0x94d049bb133111ebull;
    x ^= x >> 31;
    return x;
}

// Hash of the rows [row_lo, row_hi) of a table (a warp per row): the sum over
// entries q of row p of mix64(p << 32 | q), plus a constant for entries
// flagged one-way, p and q input indices.
__global__ void table_hash_kernel(TableArgs a, const uint32_t* __restrict__ gorig) {
    pdl_sync();
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const int nrows = 2 * a.ep->rho + 1;
    const uint16_t* const nb16 = reinterpret_cast<const uint16_t*>(a.nbr);
    unsigned long long acc = 0;
    for (uint64_t r = a.row_lo + warp; r < a.row_hi; r += nwarps) {
        const uint32_t k = (uint32_t)r;
        const unsigned long long s = a.off[k] - a.off_base, e = a.off[k + 1] - a.off_base;
        const unsigned long long p = (unsigned long long)gorig[k] << 32;
        auto add = [&](uint32_t q, bool one_way) {
            if (!VDB_GUARD(a.st, q < a.n, 17, q)) return;
            acc += mix64(p | gorig[q]) + (one_way ? 0x9e3779b97f4a7c15ull : 0ull);
        };
        if (a.compact) {
            walk_compact_row(nb16, s, e, k, a.ptile, a.tiles, a.tile_uoff, a.parts, a.trow_s,
                             a.trow_e, nrows, a.unit_words, (int)lane,
                             [&](uint32_t q, bool one_way, bool valid) {
                                 if (valid) add(q, one_way);
                             });
        } else {
            for (unsigned long long j = s + lane; j < e; j += 32) {
                const uint32_t ev = a.nbr[j];
                add(ev & kIdMask, (ev & kAsymFlag) != 0);
            }
        }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) acc += __shfl_down_sync(kFull, acc, d);
    if (lane == 0 && acc) atomicAdd(&a.st->table_hash, acc);
}

// Row chunks by one warp: each ends at the last tile whose rows still fit, found
// by a 32-way search over the row offsets (4 rounds of two dependent loads for a
// million tiles), so that the host reads a few hundred bytes of plan.  Copying
// the tiles and the n + 1 row offsets to the host for the same loop there held up
// each chunked table of 2M points by 1.4 ms.
__global__ void plan_chunks_kernel(const uint32_t* __restrict__ tiles,
                                   const uint32_t* __restrict__ ntiles,
                                   const uint32_t* __restrict__ tuoff,
                                   const unsigned long long* __restrict__ off, uint32_t n,
                                   uint64_t cap, uint32_t t0, ChunkPlan* plan) {
    pdl_sync();
    const uint32_t lane = threadIdx.x;
    const uint32_t nt = *ntiles;
    uint32_t t = t0, k = 0;
    uint32_t refused = nt > n || tiles[nt] != n ? 2u : 0u;
    while (!refused && t < nt && k < kPlanChunks) {
        const unsigned long long e0 = off[tiles[t]];
        uint32_t lo = t, hi = nt;  // the chunk's end: the last tile bound in [lo, hi] that fits
        while (lo < hi) {
            const uint64_t step = ((uint64_t)(hi - lo) + 31) / 32;
            const uint32_t probe = (uint32_t)min((uint64_t)lo + (lane + 1) * step, (uint64_t)hi);
            const uint32_t fit =
                (uint32_t)__popc(__ballot_sync(kFull, off[tiles[probe]] - e0 <= cap));
            const uint64_t base = lo;
            lo = (uint32_t)min(base + fit * step, (uint64_t)hi);
            if (fit < 32) hi = max(lo, (uint32_t)min(base + (fit + 1) * step, (uint64_t)hi) - 1u);
        }
        if (lo == t) {
            refused = 1;
        } else {
            if (lane == 0)
                plan->list[k] = RowChunk{t,         lo, tuoff[t], tuoff[lo], tiles[t], tiles[lo],
                                         e0, off[tiles[lo]]};
            k++;
            t = lo;
        }
    }
    if (lane == 0) {
        plan->n = k;
        plan->next = t;
        plan->ntiles = nt;
        plan->refused = refused;
    }
}

// Flags the table entries accepted in one direction only (the count pass
// recorded them): b in row a when dir == 1, a in row b when dir == 2.  Rows of
// 32-bit entries are sorted; of a unit's 16-bit entries those before its runs
// of whole words are (a one-way pair is never in a run).
__global__ void asym_flags_kernel(TableArgs a) {
    pdl_sync();
    uint32_t na = *a.asym_n;
    if (na > a.asym_cap) na = a.asym_cap;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < na;
         i += gridDim.x * blockDim.x) {
        const AsymPair p = a.asym[i];
        const uint32_t row = p.dir == 1u ? p.a : p.b;
        const uint32_t target = p.dir == 1u ? p.b : p.a;
        if (a.row_hi && (row < a.row_lo || row >= a.row_hi)) continue;  // row not in this chunk
        unsigned long long lo = a.off[row] - a.off_base, hi = a.off[row + 1] - a.off_base;
        const unsigned long long end = hi;
        if (a.compact) {
            // the target's position in the candidate list of the row's tile,
            // then its unit and the unit's share of the row
            const uint32_t t = a.ptile[row];
            const uint32_t slot = row - a.tiles[t];
            const uint32_t nr = 2u * (uint32_t)a.ep->rho + 1u;
            uint32_t before = 0, g = 0xffffffffu;
            for (uint32_t i = 0; i < nr; i++) {
                const unsigned long long k = (unsigned long long)t * nr + i;
                const uint32_t s0 = a.trow_s[k], e0 = a.trow_e[k];
                if (target >= s0 && target < e0) g = before + (target - s0);
                before += e0 - s0;
            }
            const uint32_t u0 = a.tile_uoff[t], nu = a.tile_uoff[t + 1] - u0;
            const uint32_t c = g / (a.unit_words * 32u), pos = g % (a.unit_words * 32u);
            if (!VDB_GUARD(a.st, g != 0xffffffffu && c < max(nu, 1u) && slot < kUnitQ, 5, target))
                continue;
            if (nu) {  // (a small tile's row is one piece)
                for (uint32_t u = u0; u < u0 + c; u++)
                    lo += a.parts[(unsigned long long)u * kUnitQ + slot];
                // (a one-way pair was tested: it is not in the runs that follow the
                // unit's other entries)
                uint32_t in_runs = 0;
                if (a.wflags)
                    for (uint32_t b = 0; b < flag_blocks(a.unit_words); b++)
                        in_runs += 32u * (uint32_t)__popc(full_runs(
                                             a.wflags[(unsigned long long)(u0 + c) * flag_blocks(a.unit_words) + b].x,
                                             c * a.unit_words + 32u * b, before));
                hi = lo + a.parts[(unsigned long long)(u0 + c) * kUnitQ + slot] - in_runs;
            }
            if (hi > end) hi = end;
            if (lo > hi) lo = hi;
            const unsigned long long seg_end = hi;
            uint16_t* const nb = reinterpret_cast<uint16_t*>(a.nbr);
            while (lo < hi) {
                const unsigned long long mid = (lo + hi) >> 1;
                if ((uint32_t)(nb[mid] & kPosMask16) < pos) lo = mid + 1;
                else hi = mid;
            }
            if (VDB_GUARD(a.st, lo < seg_end && (uint32_t)(nb[lo] & kPosMask16) == pos,
                          5, target))
                nb[lo] |= kAsymFlag16;
            continue;
        }
        while (lo < hi) {
            const unsigned long long mid = (lo + hi) >> 1;
            if ((a.nbr[mid] & kIdMask) < target) lo = mid + 1;
            else hi = mid;
        }
        if (VDB_GUARD(a.st, lo < end && (a.nbr[lo] & kIdMask) == target, 5, target))
            a.nbr[lo] |= kAsymFlag;
    }
}

}  // namespace
int table_block_threads() { return kTT; }
// tiles hold at most one warp tile of queries (the count and table passes
// give each warp one tile; the fill pass's blocks accept up to kTT * kQPT)
int table_tile_queries() {
    static_assert(kWQ <= kTT * kQPT, "fill blocks must hold a whole tile");
    return kWQ;
}

void launch_count(const TableArgs& a, int nblocks, cudaStream_t s) {
    if (!a.mixed || a.n > kSmallFused) {
        const unsigned nb = (a.n + kTT - 1) / kTT;
        if (a.mixed)
            launch(small_count_kernel<true>, nb, kTT, s, a);
        else
            launch(small_count_kernel<false>, nb, kTT, s, a);
    }
    if (a.mixed)
        launch(count_kernel<true>, nblocks, kWPB * 32, s, a);
    else
        launch(count_kernel<false>, nblocks, kWPB * 32, s, a);
}

void launch_fill(const TableArgs& a, int nblocks, cudaStream_t s) {
    if (a.mixed)
        launch(fill_kernel<true>, nblocks, kTT, s, a);
    else
        launch(fill_kernel<false>, nblocks, kTT, s, a);
}

size_t words_state_bytes(uint32_t n) {
    return 2 * ((look_state_bytes(((uint64_t)n + kLookThreads - 1) / kLookThreads) + 15) & ~(size_t)15);
}

void launch_tile_words(const TableArgs& a, unsigned long long* boff, uint32_t* uoff,
                       unsigned long long* nwords, uint32_t* nunits, void* zeroed,
                       cudaStream_t s) {
    if (!a.n) return;
    const unsigned nb = (a.n + kLookThreads - 1) / kLookThreads;
    launch(tile_words_kernel, nb, kLookThreads, s, a, boff, uoff, nwords, nunits, look_state(zeroed),
        look_state((char*)zeroed + words_state_bytes(a.n) / 2));
}

void launch_unit_list(const TableArgs& a, uint32_t* ulist, cudaStream_t s) {
    if (!a.n) return;
    const uint32_t boxes = a.wbox ? ((a.n + 3u) / 4u + kTT - 1) / kTT : 0u;
    launch(unit_list_kernel, boxes + (a.n + kTT - 1) / kTT, kTT, s, a, ulist, boxes);
}

void launch_expand(const TableArgs& a, int nblocks, cudaStream_t s) {
    if (a.n > kSmallFused && a.row_hi > a.row_lo) {
        const unsigned nb = (a.row_hi - a.row_lo + kTT - 1) / kTT;
        if (a.compact)
            launch(small_expand_kernel<uint16_t>, nb, kTT, s, a);
        else
            launch(small_expand_kernel<uint32_t>, nb, kTT, s, a);
    }
    if (a.unit_hi <= a.unit_lo && a.n > kSmallFused) return;
    if (a.compact)
        launch(expand16_kernel, nblocks, kXPB * 32, s, a);
    else
        launch(expand_kernel<uint32_t>, nblocks, kXPB * 32, s, a);
}

void launch_table_hash(const TableArgs& a, const uint32_t* gorig, int nblocks, cudaStream_t s) {
    if (a.row_hi <= a.row_lo) return;
    launch(table_hash_kernel, nblocks, kTT, s, a, gorig);
}

void launch_asym_flags(const TableArgs& a, cudaStream_t s) {
    launch(asym_flags_kernel, 64, kTT, s, a);
}

void launch_plan_chunks(const uint32_t* tiles, const uint32_t* ntiles, const uint32_t* tuoff,
                        const unsigned long long* off, uint32_t n, uint64_t cap, uint32_t t0,
                        ChunkPlan* plan, cudaStream_t s) {
    launch(plan_chunks_kernel, 1, 32, s, tiles, ntiles, tuoff, off, n, cap, t0, plan);
}

int table_blocks_per_sm(bool fill, bool mixed) {
    int nb = 0;
    if (fill) {
        if (mixed)
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fill_kernel<true>, kTT, 0);
        else
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fill_kernel<false>, kTT, 0);
    } else {
        if (mixed)
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, count_kernel<true>, kWPB * 32, 0);
        else
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, count_kernel<false>, kWPB * 32, 0);
    }
    return nb > 0 ? nb : 1;
}

int expand_blocks_per_sm(bool compact) {
    int nb = 0;
    if (compact)
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, expand16_kernel, kXPB * 32, 0);
    else
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, expand_kernel<uint32_t>, kXPB * 32, 0);
    return nb > 0 ? nb : 1;
}

}  // namespace vdb
