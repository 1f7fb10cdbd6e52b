// Index construction on the device:
//  * the reference's visit order (binDataset, src/main.cpp:459-605),
//  * its multiple-point boxes (createEntryMBBMultiplePoints, src/main.cpp:404-436;
//    MPBRect::CreateMBB, src/structs.h:79-120),
//  * the uniform grid that replaces its R-tree for candidate generation:
//    cell keys, cell-ordered coordinates, cell start offsets and query tiles.
#include <float.h>

#include "vdb_lookback.cuh"

namespace vdb {

namespace {

constexpr int kThreads = 256;

inline unsigned nblk(uint64_t n) { return (unsigned)((n + kThreads - 1) / kThreads); }

// Digit counts of a key in shared memory, added to the sort's histogram at
// the end of the block.
struct DigitCounts {
    uint32_t c[kMaxPasses][kDigits];
};
__device__ __forceinline__ void counts_clear(DigitCounts& h, int passes) {
    for (uint32_t i = threadIdx.x; i < (uint32_t)passes * kDigits; i += blockDim.x)
        (&h.c[0][0])[i] = 0u;
    __syncthreads();
}
__device__ __forceinline__ void counts_add(DigitCounts& h, int passes, uint32_t key) {
    for (int p = 0; p < passes; p++)
        atomicAdd(&h.c[p][(key >> (p * kDigitBits)) & (kDigits - 1u)], 1u);
}
__device__ __forceinline__ void counts_flush(DigitCounts& h, int passes, uint32_t* hist) {
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < (uint32_t)passes * kDigits; i += blockDim.x) {
        const uint32_t v = (&h.c[0][0])[i];
        if (v) atomicAdd(&hist[i], v);
    }
}

// floor(r) of a quotient that FP32 knows as r, within err: exact wherever r is
// further than err from a whole number; *sure = 0 otherwise (and for NaN and
// infinities), and the caller divides in FP64.  GB300 issues 2 FP64 lanes a
// cycle per SM, and two divisions per point bounded the key kernels (1M
// points: 54 us; 13 us with the filter).
__device__ __forceinline__ float floor_if_sure(float r, float err, bool* sure) {
    const float f = floorf(r);
    *sure = r - f > err && r - f < 1.0f - err;
    return f;
}
// usable FP32 factor (1 / w and 300 / w stay far from FP32's limits)
__device__ __forceinline__ bool factor_ok(float v) { return v > 1e-30f && v < 1e30f; }

// Bin key of src/main.cpp:491-540 with the same FP64 results:
// width = (max-min)*1.01, offset = -min (or fabs(min)), bin = floor(((x+offset)/width)*300).
// The FP32 quotient is off by less than 4 * 2^-24 of itself (conversion,
// factor, product; the FP64 roundings of the exact sequence are far smaller),
// which is below 1e-4 of a bin for bins up to 300; 1e-3 is required.
__global__ void __launch_bounds__(kThreads) visit_keys_kernel(
    const double* __restrict__ x, const double* __restrict__ y, uint32_t n,
    const BBox* __restrict__ bb, uint32_t* __restrict__ keys, int passes,
    uint32_t* __restrict__ hist, DeviceStatus* st) {
    pdl_sync();
    __shared__ DigitCounts s_h;
    __shared__ double s_p[4];
    __shared__ float s_f[2];
    if (threadIdx.x < 2) {
        const double mn = threadIdx.x ? bb->miny : bb->minx, mx = threadIdx.x ? bb->maxy : bb->maxx;
        const double w = __dmul_rn(__dsub_rn(mx, mn), 1.01);
        s_p[threadIdx.x] = w;
        s_p[2 + threadIdx.x] = (mn > 0) ? -mn : fabs(mn);
        s_f[threadIdx.x] = (float)((double)kVisitBins / w);
    }
    counts_clear(s_h, passes);
    // (bins as integers: compared and converted as doubles they took 26 us of the
    // FP64 pipe's time at 2M points, 7 at 1M)
    constexpr uint32_t kNoBin = 0xffffffffu;
    auto bin = [&](double v, int axis) -> uint32_t {
        const double a = __dadd_rn(v, s_p[2 + axis]);
        const float r = (float)a * s_f[axis];
        bool sure;
        const float f = floor_if_sure(r, 1e-3f, &sure);
        if (sure && factor_ok(s_f[axis]) && f >= 0.0f && f <= (float)(kVisitBins - 1))
            return (uint32_t)f;
        const double b = floor(__dmul_rn(__ddiv_rn(a, s_p[axis]), (double)kVisitBins));
        return b >= 0.0 && b <= (double)(kVisitBins - 1) ? (uint32_t)b : kNoBin;
    };
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t bx = bin(x[i], 0), by = bin(y[i], 1);
        if (bx == kNoBin || by == kNoBin) {
            atomicOr(&st->flags, kStatDegenerate);
            bx = 0;
            by = 0;
        }
        const uint32_t key = bx * kVisitBins + by;
        keys[i] = key;
        counts_add(s_h, passes, key);
    }
    counts_flush(s_h, passes, hist);
}

// One warp per box: the bounding box of visit positions [b*mbb, b*mbb+mbb)
// (the lanes gather the box's points 32 at a time, then reduce).
__global__ void mpb_kernel(const double* __restrict__ x, const double* __restrict__ y,
                           const uint32_t* __restrict__ vorder, uint32_t n, int mbb,
                           uint32_t nboxes, MpbBox* __restrict__ boxes) {
    pdl_sync();
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t b = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (b >= nboxes) return;  // (whole warps)
    const uint64_t s = b * (uint32_t)mbb;
    uint64_t e = s + (uint32_t)mbb;
    if (e > n) e = n;
    // (ordered keys; a minimum is the complement of the complements' maximum)
    unsigned long long x0 = 0, x1 = 0, y0 = 0, y1 = 0;
#pragma unroll 2
    for (uint64_t k = s + lane; k < e; k += 32) {
        const uint32_t o = vorder[k];
        const unsigned long long kx = ordered_key(x[o]), ky = ordered_key(y[o]);
        x0 = max(x0, ~kx);
        x1 = max(x1, kx);
        y0 = max(y0, ~ky);
        y1 = max(y1, ky);
    }
    x0 = warp_max_u64(x0);
    x1 = warp_max_u64(x1);
    y0 = warp_max_u64(y0);
    y1 = warp_max_u64(y1);
    if (lane == 0)
        boxes[b] = MpbBox{ordered_value(~x0), ordered_value(x1), ordered_value(~y0),
                          ordered_value(y1)};
}

// Cell of v, floor((v - v0) / w) in FP64, and its subcell (of 2^sub per cell),
// which only orders the points of a cell.  FP32 decides where its quotient,
// off by less than 4 * 2^-24 of itself, is surely between two whole numbers.
__device__ __forceinline__ uint32_t cell_of(double v, double v0, double w, float iw, uint32_t nc,
                                            uint32_t sub, uint32_t* sc) {
    const double a = __dsub_rn(v, v0);
    const float r = (float)a * iw;
    bool sure;
    float f32 = floor_if_sure(r, 4e-7f * r + 1e-6f, &sure);
    const float subs = (float)(1u << sub);
    if (sure && factor_ok(iw) && f32 >= 0.0f && f32 < 8388608.0f && (uint32_t)f32 < nc) {
        *sc = (uint32_t)fminf((r - f32) * subs, subs - 1.0f);
        return (uint32_t)f32;
    }
    const double q = __ddiv_rn(a, w);
    double f = floor(q);
    if (!(f >= 0.0)) f = 0.0;
    if (f > (double)(nc - 1)) f = (double)(nc - 1);
    *sc = (uint32_t)fminf(fmaxf((float)(q - f) * subs, 0.f), subs - 1.0f);
    return (uint32_t)f;
}

// Place of subcell (x, y) along the Hilbert curve over 2^sub x 2^sub subcells:
// from the coarsest quadrant down, each level turned the way the curve enters
// it (the textbook walk over quadrants, after Hilbert 1891).  Every run of the curve is connected, so a run of points has a small box
// (along the Z order every second step is a diagonal or a jump).
__device__ __forceinline__ uint32_t curve_index(uint32_t x, uint32_t y, uint32_t sub) {
    uint32_t d = 0;
    for (int b = (int)sub - 1; b >= 0; b--) {
        const uint32_t rx = (x >> b) & 1u, ry = (y >> b) & 1u;
        d = (d << 2) | ((3u * rx) ^ ry);
        if (!ry) {
            if (rx) {
                x = ~x;
                y = ~y;
            }
            const uint32_t t = x;
            x = y;
            y = t;
        }
    }
    return d;
}

__global__ void __launch_bounds__(kThreads) grid_keys_kernel(
    const double* __restrict__ x, const double* __restrict__ y, uint32_t n, GridParams g,
    uint32_t* __restrict__ keys, int passes, uint32_t* __restrict__ hist, EpsParams ep,
    EpsParams* __restrict__ ep_out) {
    pdl_sync();
    __shared__ DigitCounts s_h;
    counts_clear(s_h, passes);
    if (blockIdx.x == 0 && threadIdx.x == 0) *ep_out = ep;
    const float iw = ep.iw;  // (an FP64 division by each thread took 2 us of 25 at 1M points)
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t sx = 0, sy = 0;
        const uint32_t cx = cell_of(x[i], g.x0, g.w, iw, g.ncx, g.sub, &sx);
        const uint32_t cy = cell_of(y[i], g.y0, g.w, iw, g.ncy, g.sub, &sy);
        uint32_t key = cy * g.ncx_pad + cx;
        key = (key << (2u * g.sub)) | curve_index(sx, sy, g.sub);
        keys[i] = key;
        counts_add(s_h, passes, key);
    }
    counts_flush(s_h, passes, hist);
}

// Cell-ordered copies of point k: FP64 coordinates, FP32 coordinates relative
// to the own cell's origin (the FP64 shift is exact up to one rounding; the
// FP32 conversion adds one more), visit position and multiple-point box.
__device__ __forceinline__ void gather_point(const OrderArgs& a, uint32_t k, uint32_t key) {
    const uint32_t o = a.gorig[k];
    const double xv = a.x[o], yv = a.y[o];
    const uint32_t cy = key / a.g.ncx_pad, cx = key - cy * a.g.ncx_pad;
    const double ox = __dadd_rn(a.g.x0, __dmul_rn((double)cx, a.g.w));
    const double oy = __dadd_rn(a.g.y0, __dmul_rn((double)cy, a.g.w));
    a.gxy[k] = make_double2(xv, yv);
    a.glocal[k] = make_float2(__double2float_rn(__dsub_rn(xv, ox)),
                              __double2float_rn(__dsub_rn(yv, oy)));
    const uint32_t p = a.pos[o];
    a.gpos[k] = p;
    a.gbox[k] = a.mpb[p / a.mbb];
}

__global__ void gather_kernel(OrderArgs a) {
    pdl_sync();
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < a.n) gather_point(a, k, k);
}

// One pass over the sorted keys: the gathers, and the first points of cells
// and tiles compacted by a single-pass scan (both counts in one state word, 31
// bits each).  A warp takes 32 * kOrderItems consecutive points.  The tiles of a
// group of cells start every tq points from the group's first point (found by
// looking back for the last group start): cut at multiples of tq of the point
// index instead, a cell of 30 points was two tiles half of the time.
constexpr int kOrderItems = 2;
constexpr uint32_t kOrderTile = kLookThreads * kOrderItems;
__global__ void __launch_bounds__(kLookThreads) order_kernel(OrderArgs a, LookState ls,
                                                             unsigned long long* marks) {
    pdl_sync();
    __shared__ uint32_t s_last[kLookThreads / 32];  // 1 + the warp's last group start, or 0
    __shared__ uint32_t s_in;
    const uint32_t tile = lookback_ticket(ls);
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint64_t base = (uint64_t)tile * kOrderTile + wid * (32u * kOrderItems);
    uint32_t key[kOrderItems], bc[kOrderItems], bt[kOrderItems];
    uint32_t last = 0;
#pragma unroll
    for (int i = 0; i < kOrderItems; i++) {
        const uint64_t k = base + 32u * i + lane;
        const bool in = k < a.n;
        key[i] = in ? a.gkey[k] : 0u;
        uint32_t prev = __shfl_up_sync(0xffffffffu, key[i], 1);
        if (lane == 0 && in && k > 0) prev = a.gkey[k - 1];
        bc[i] = __ballot_sync(0xffffffffu, in && (k == 0 || key[i] != prev));
        bt[i] = __ballot_sync(0xffffffffu, in && (k == 0 || key[i] / a.g.G != prev / a.g.G));
        if (bt[i]) last = (uint32_t)base + 32u * i + 32u - (uint32_t)__clz((int)bt[i]);
    }
    if (lane == 0) s_last[wid] = last;
    __syncthreads();
    if (wid == 0) {
        uint32_t mine = lane < kLookThreads / 32 ? s_last[lane] : 0u;
        mine = __reduce_max_sync(0xffffffffu, mine);
        const uint32_t in = (uint32_t)warp_last_mark(mine, tile, marks, a.st);
        if (lane == 0) s_in = in;
    }
    __syncthreads();
    uint32_t start = s_in;
    for (uint32_t w = 0; w < wid; w++) start = max(start, s_last[w]);
    unsigned long long mine = 0;  // cells | tiles << 31 of the warp
#pragma unroll
    for (int i = 0; i < kOrderItems; i++) {
        const uint64_t k = base + 32u * i + lane;
        const uint32_t upto = bt[i] & ((2u << lane) - 1u);
        const uint32_t s1 = upto ? (uint32_t)base + 32u * i + 32u - (uint32_t)__clz((int)upto) : start;
        if (bt[i]) start = (uint32_t)base + 32u * i + 32u - (uint32_t)__clz((int)bt[i]);
        bt[i] = __ballot_sync(0xffffffffu, k < a.n && ((uint32_t)k + 1u - s1) % a.tq == 0u);
        mine += (unsigned long long)__popc(bc[i]) | ((unsigned long long)__popc(bt[i]) << 31);
    }
    const unsigned long long before = block_lookback(lane == 31 ? mine : 0ull, tile, ls, a.st);
    uint32_t c0 = (uint32_t)(before & 0x7fffffffull), t0 = (uint32_t)(before >> 31);
    const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
    for (int i = 0; i < kOrderItems; i++) {
        const uint64_t k64 = base + 32u * i + lane;
        const uint32_t k = (uint32_t)k64;
        if (k64 < a.n) {
            const uint32_t c = c0 + __popc(bc[i] & lt), t = t0 + __popc(bt[i] & lt);
            const uint32_t fc = (bc[i] >> lane) & 1u, ft = (bt[i] >> lane) & 1u;
            if (!VDB_GUARD(a.st, c + fc <= a.n && t + ft <= a.n && t + ft > 0u, 19, c)) return;
            a.cscan[k] = c;
            if (fc) {
                a.clist[c] = k;
                a.ckey[c] = key[i];
                a.ccx[c] = key[i] % a.g.ncx_pad;
            }
            if (ft) a.tiles[t] = k;
            a.ptile[k] = t + ft - 1u;
            if (k == a.n - 1) {
                a.cscan[a.n] = c + fc;
                a.clist[c + fc] = a.n;
                a.tiles[t + ft] = a.n;
                *a.ntiles = t + ft;
            }
            if (a.cbest) a.cbest[k] = 0ull;
            gather_point(a, k, key[i]);
        }
        c0 += __popc(bc[i]);
        t0 += __popc(bt[i]);
    }
}

// First cell of ckey[0..ncl) with a key >= v: 33-ary search by a warp.
__device__ __forceinline__ uint32_t warp_lower_bound(const uint32_t* __restrict__ ckey,
                                                     uint32_t ncl, uint64_t v) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t lo = 0, hi = ncl;
    while (hi > lo) {
        const uint32_t len = hi - lo;
        // probes lo + (len * (lane + 1)) / 33 are increasing and below hi
        const uint32_t p = lo + (uint32_t)(((uint64_t)len * (lane + 1)) / 33u);
        const uint32_t below = __ballot_sync(0xffffffffu, (uint64_t)ckey[p] < v);
        const uint32_t nb = __popc(below);
        if (nb < 32) hi = __shfl_sync(0xffffffffu, p, (int)nb);
        if (nb > 0) lo = __shfl_sync(0xffffffffu, p, (int)nb - 1) + 1u;
    }
    return lo;
}

// Dense cell array, one block per kFillCells keys: the block finds its cells
// among the sorted non-empty ones, drops their first points into shared memory
// and fills every gap with the next cell's by a suffix minimum.  Each entry is
// written once (26M cells: 31 us; memset, marks and a three-kernel suffix scan
// took 170).
constexpr int kFillItems = 16;
constexpr uint32_t kFillCells = kThreads * kFillItems;
__global__ void __launch_bounds__(kThreads) cell_start_kernel(const uint32_t* __restrict__ ckey,
                                                              const uint32_t* __restrict__ clist,
                                                              const uint32_t* __restrict__ nclp,
                                                              uint32_t n, uint64_t entries,
                                                              uint32_t* __restrict__ cell_start) {
    pdl_sync();
    __shared__ uint32_t s_v[kFillCells + kFillCells / kFillItems];  // 16 cells and a pad word
    __shared__ uint32_t s_lim[2], s_warp[kThreads / 32];
    const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const uint64_t c0 = (uint64_t)blockIdx.x * kFillCells;
    const uint32_t ncl = *nclp;
    if (wid < 2) {
        const uint32_t b = warp_lower_bound(ckey, ncl, c0 + (wid ? kFillCells : 0u));
        if (lane == 0) s_lim[wid] = b;
    }
    for (uint32_t i = tid; i < kFillCells + kFillCells / kFillItems; i += kThreads)
        s_v[i] = 0xffffffffu;
    __syncthreads();
    const uint32_t lo = s_lim[0], hi = s_lim[1];
    const uint32_t next = hi < ncl ? clist[hi] : n;
    if (lo < hi) {
        for (uint32_t i = lo + tid; i < hi; i += kThreads) {
            const uint32_t j = (uint32_t)(ckey[i] - c0);
            s_v[j + j / kFillItems] = clist[i];
        }
        __syncthreads();
        uint32_t* mine = s_v + tid * (kFillItems + 1);
        uint32_t m = 0xffffffffu;
#pragma unroll
        for (int i = 0; i < kFillItems; i++) m = min(m, mine[i]);
        // smallest value after this thread's cells (first points ascend)
        uint32_t suf = m;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t o = __shfl_down_sync(0xffffffffu, suf, d);
            if (lane + d < 32u) suf = min(suf, o);
        }
        if (lane == 0) s_warp[wid] = suf;
        __syncthreads();
        uint32_t after = __shfl_down_sync(0xffffffffu, suf, 1);
        if (lane == 31) after = 0xffffffffu;
        for (uint32_t w = wid + 1; w < kThreads / 32; w++) after = min(after, s_warp[w]);
        after = min(after, next);
#pragma unroll
        for (int i = kFillItems - 1; i >= 0; i--) {
            after = min(after, mine[i]);
            mine[i] = after;
        }
        __syncthreads();
        for (uint32_t i = tid; i < kFillCells; i += kThreads)
            if (c0 + i < entries) cell_start[c0 + i] = s_v[i + i / kFillItems];
    } else {
        for (uint32_t i = tid; i < kFillCells; i += kThreads)
            if (c0 + i < entries) cell_start[c0 + i] = next;
    }
}

__global__ void cell_rows_kernel(const uint32_t* __restrict__ ckey,
                                 const uint32_t* __restrict__ nclp, uint32_t ncx_pad, uint32_t ncy,
                                 uint32_t* __restrict__ crow) {
    pdl_sync();
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r > ncy) return;
    const uint64_t v = (uint64_t)r * ncx_pad;
    uint32_t b = 0, e = *nclp;
    while (b < e) {
        const uint32_t m = (b + e) >> 1;
        if ((uint64_t)ckey[m] < v) b = m + 1;
        else e = m;
    }
    crow[r] = b;
}

}  // namespace

// Blocks of the key kernels: enough to fill the chip, and for large inputs
// few enough that adding the digit counts up costs little.
unsigned key_blocks(uint32_t n) { return std::min<unsigned>(nblk(n), 152u * 8u); }

void launch_visit_keys(const double* x, const double* y, uint32_t n, const BBox* bb,
                       uint32_t* keys, uint32_t* hist, DeviceStatus* st, cudaStream_t s) {
    if (!n) return;
    launch(visit_keys_kernel, key_blocks(n), kThreads, s, x, y, n, bb, keys, sort_passes(kVisitBits),
                                                         hist, st);
}

void launch_mpb_boxes(const double* x, const double* y, const uint32_t* vorder, uint32_t n,
                      int mbb, MpbBox* boxes, cudaStream_t s) {
    uint32_t nb = (uint32_t)(((uint64_t)n + (uint32_t)mbb - 1) / (uint32_t)mbb);
    if (nb) {
        launch(mpb_kernel, nblk((uint64_t)nb * 32u), kThreads, s, x, y, vorder, n, mbb, nb,
                                                                  boxes);
    }
}

void launch_grid_keys(const double* x, const double* y, uint32_t n, GridParams g, int bits,
                      uint32_t* keys, uint32_t* hist, const EpsParams& ep, EpsParams* ep_out,
                      cudaStream_t s) {
    if (!n) return;
    launch(grid_keys_kernel, key_blocks(n), kThreads, s, x, y, n, g, keys, sort_passes(bits), hist,
           ep, ep_out);
}

size_t order_state_bytes(uint32_t n) {
    const uint64_t nb = ((uint64_t)n + kOrderTile - 1) / kOrderTile;
    return look_state_bytes(nb) + nb * 8;
}

void launch_order(const OrderArgs& a, void* zeroed, cudaStream_t s) {
    if (!a.n) return;
    const unsigned nb = (unsigned)(((uint64_t)a.n + kOrderTile - 1) / kOrderTile);
    launch(order_kernel, nb, kLookThreads, s, a, look_state(zeroed),
           (unsigned long long*)((char*)zeroed + look_state_bytes(nb)));
}

void launch_gather(const OrderArgs& a, cudaStream_t s) {
    if (!a.n) return;
    launch(gather_kernel, nblk(a.n), kThreads, s, a);
}

void launch_cell_start(const uint32_t* ckey, const uint32_t* clist, const uint32_t* ncl,
                       uint32_t n, const GridParams& g, uint32_t* cell_start, cudaStream_t s) {
    const uint64_t entries = g.ncells + 1;
    launch(cell_start_kernel, (unsigned)((entries + kFillCells - 1) / kFillCells), kThreads, s, ckey, clist, ncl, n, entries, cell_start);
}

void launch_cell_rows(const uint32_t* ckey, const uint32_t* ncl, const GridParams& g,
                      uint32_t* crow, cudaStream_t s) {
    launch(cell_rows_kernel, nblk((uint64_t)g.ncy + 1), kThreads, s, ckey, ncl, g.ncx_pad, g.ncy,
                                                                   crow);
}

}  // namespace vdb
