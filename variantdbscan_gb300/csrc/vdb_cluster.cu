// Cluster labelling from the neighbour table, reproducing the labels of the
// reference's sequential expansion (DBScan::algDBScanParallel,
// src/DBScan.cpp:523-609) without running it sequentially.
//
// With pos(p) the reference's visit position (binDataset order):
//   core(p)   <=> |N(p)| >= minpts (N(p) contains p);
//   components of the core points under the symmetric core-core edges are
//   found by lock-free union-find (link the larger root under the smaller);
//   seed(C) = min pos over the cores of C.  The reference's main loop reaches
//   the cores of C first at seed(C) and its expansion then visits every point
//   reachable from C, so a cluster starts at seed(C) and numbers follow seeds.
//   A core-core edge accepted in one direction only (the R-tree box rule,
//   see vdb_table.cu) lets the cluster started by one component absorb
//   another; resolve_kernel replays that on the component graph in seed order.
//   A non-core point p joins the cluster with the earliest start among the
//   cores u with p in N(u), if that start precedes pos(p); otherwise the main
//   loop visited p first and labelled it noise (src/DBScan.cpp:552-554,
//   573-577).
#include <algorithm>

#include "vdb_internal.cuh"

namespace vdb {

namespace {

constexpr int kThreads = 256;
constexpr uint32_t kNone = 0xffffffffu;
constexpr unsigned kFull = 0xffffffffu;

inline unsigned nblk(uint64_t n) { return (unsigned)((n + kThreads - 1) / kThreads); }

__device__ __forceinline__ bool is_core(uint32_t d, unsigned long long minpts) {
    return (unsigned long long)d >= minpts;
}

// Root of x.  Ends after at most x steps: every parent is at most its child
// (unions link the larger root under the smaller one, path halving stores an
// ancestor), so the chain strictly decreases until it meets a root.
__device__ __forceinline__ uint32_t uf_find(uint32_t* parent, uint32_t x) {
    volatile uint32_t* vp = parent;
    uint32_t p = vp[x];
    while (p != x) {
        const uint32_t gp = vp[p];
        if (gp != p) vp[x] = gp;  // path halving; parents only decrease
        x = p;
        p = gp;
    }
    return x;
}

__device__ __forceinline__ void uf_union(uint32_t* parent, uint32_t a, uint32_t b,
                                         DeviceStatus* st) {
    for (int it = 0; it < (1 << 24); it++) {
        a = uf_find(parent, a);
        b = uf_find(parent, b);
        if (a == b) return;
        if (a > b) {
            const uint32_t t = a;
            a = b;
            b = t;
        }
        const uint32_t old = atomicCAS(&parent[b], b, a);
        if (old == b) return;
        b = old;
    }
    atomicOr(&st->flags, kStatUnionStall);
}

__global__ void uf_init_kernel(ClusterArgs a, int fresh) {
    pdl_sync();
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < a.nw) a.bits[k] = 0u;
    if (k >= a.n) return;
    if (fresh) a.parent[k] = k;
    a.seed[k] = kNone;
    a.best[k] = kNone;
    a.cstart[k] = k;
}

// One warp per row.  From scratch, an edge (k, v) of two cores is united from
// its smaller end; when the parent array already holds the components of a
// larger minpts, only rows of the new cores are read and all their core
// neighbours are united.
__global__ void uf_union_kernel(ClusterArgs a) {
    pdl_sync();
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const bool reuse = a.minpts_prev != ~0ull;
    for (uint64_t r = a.row_lo + warp; r < a.row_hi; r += nwarps) {
        const uint32_t k = (uint32_t)r;
        const uint32_t dk = a.deg[k];
        if (!is_core(dk, a.minpts)) continue;
        if (reuse && is_core(dk, a.minpts_prev)) continue;
        const unsigned long long s = a.off[k] - a.off_base, e = a.off[k + 1] - a.off_base;
        auto edge = [&](uint32_t v) {
            if (!VDB_GUARD(a.st, v < a.n, 10, v)) return;
            if (v == k || (!reuse && v < k)) return;
            if (!is_core(a.deg[v], a.minpts)) return;
            uf_union(a.parent, k, v, a.st);
        };
        if (a.compact) {
            walk_compact_row(reinterpret_cast<const uint16_t*>(a.nbr), s, e, k, a.ptile, a.tiles,
                             a.tile_uoff, a.parts, a.trow_s, a.trow_e, 2 * a.ep->rho + 1,
                             a.unit_words, (int)lane, [&](uint32_t v, bool one_way, bool valid) {
                                 if (valid && !one_way) edge(v);
                             });
        } else {
            for (unsigned long long j = s + lane; j < e; j += 32) {
                const uint32_t ev = a.nbr[j];
                if (!(ev & kAsymFlag)) edge(ev & kIdMask);
            }
        }
    }
}

// Read-only find: while the flatten pass stores roots, a path-halving write of
// another thread could replace a stored root by an intermediate ancestor.
__device__ __forceinline__ uint32_t uf_find_ro(const uint32_t* parent, uint32_t x) {
    const volatile uint32_t* vp = parent;
    uint32_t p = vp[x];
    while (p != x) {
        x = p;
        p = vp[x];
    }
    return x;
}

__global__ void save_components_kernel(ClusterArgs a, uint32_t* __restrict__ comp) {
    pdl_sync();
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= a.n) return;
    const uint32_t p = a.gpos[k];
    if (!VDB_GUARD(a.st, p < a.n, 18, p)) return;
    comp[p] = is_core(a.deg[k], a.minpts) ? a.seed[a.parent[k]] : kNone;
}

__global__ void uf_flatten_kernel(ClusterArgs a) {
    pdl_sync();
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= a.n || !is_core(a.deg[k], a.minpts)) return;
    const uint32_t r = uf_find_ro(a.parent, k);
    a.parent[k] = r;
    // cell-ordered neighbours mostly share a root: one atomic per root and warp
    const uint32_t same = __match_any_sync(__activemask(), r);
    const uint32_t mn = __reduce_min_sync(same, a.gpos[k]);
    if ((threadIdx.x & 31) == (uint32_t)(__ffs(same) - 1)) atomicMin(&a.seed[r], mn);
}

// Directed core-core edges between different components (single thread; the
// list is empty unless the box rule broke the symmetry of a core pair).
__global__ void resolve_kernel(ClusterArgs a, uint32_t* ws, uint32_t cap) {
    pdl_sync();
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    uint32_t na = *a.asym_count;
    if (na > a.asym_cap) na = a.asym_cap;
    uint32_t* efrom = ws;
    uint32_t* eto = ws + cap;
    uint32_t* nodes = ws + 2 * cap;
    uint32_t* stack = ws + 4 * cap;  // 2*cap entries
    uint32_t ne = 0;
    for (uint32_t i = 0; i < na; i++) {
        const AsymPair p = a.asym[i];
        if (!is_core(a.deg[p.a], a.minpts) || !is_core(a.deg[p.b], a.minpts)) continue;
        const uint32_t ra = a.parent[p.a], rb = a.parent[p.b];
        if (ra == rb) continue;
        if (ne >= cap) {
            atomicOr(&a.st->flags, kStatResolveOverflow);
            return;
        }
        if (p.dir == 1u) {  // b in N(a) only: a's expansion reaches b
            efrom[ne] = ra;
            eto[ne] = rb;
        } else {
            efrom[ne] = rb;
            eto[ne] = ra;
        }
        ne++;
    }
    if (ne == 0) return;
    // distinct endpoint components in seed order
    uint32_t nn = 0;
    for (uint32_t i = 0; i < 2 * ne; i++) {
        const uint32_t r = i < ne ? efrom[i] : eto[i - ne];
        bool dup = false;
        for (uint32_t j = 0; j < nn && !dup; j++) dup = nodes[j] == r;
        if (dup) continue;
        uint32_t j = nn++;
        while (j > 0 && a.seed[nodes[j - 1]] > a.seed[r]) {
            nodes[j] = nodes[j - 1];
            j--;
        }
        nodes[j] = r;
    }
    for (uint32_t i = 0; i < nn; i++) a.cstart[nodes[i]] = kNone;
    for (uint32_t i = 0; i < nn; i++) {
        const uint32_t u = nodes[i];
        if (a.cstart[u] != kNone) continue;
        a.cstart[u] = u;
        uint32_t top = 0;
        stack[top++] = u;
        while (top) {
            const uint32_t x = stack[--top];
            for (uint32_t e = 0; e < ne; e++) {
                if (efrom[e] != x) continue;
                const uint32_t y = eto[e];
                if (a.cstart[y] != kNone) continue;
                a.cstart[y] = u;
                stack[top++] = y;
            }
        }
    }
}

// Cluster numbers: a cluster's number is the rank of its start among the
// starts (visit positions, one bit each).  rank[w] = starts before word w;
// returns their number (one block; nw: start_words).
constexpr int kRankThreads = 1024;
constexpr int kRankItems = 8;
__device__ uint32_t rank_bits(const uint32_t* bits, uint32_t* __restrict__ rank, uint32_t nw) {
    __shared__ uint32_t s_tot[32];
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t carry = 0;
    for (uint32_t base = 0; base < nw; base += kRankThreads * kRankItems) {
        const uint32_t w0 = base + threadIdx.x * kRankItems;
        uint32_t c[kRankItems], sum = 0;
        uint4 lo = make_uint4(0, 0, 0, 0), hi = lo;
        if (w0 < nw) {  // (nw is a multiple of kRankItems)
            // (from L2: other blocks of this kernel may have set them)
            lo = __ldcg(reinterpret_cast<const uint4*>(bits + w0));
            hi = __ldcg(reinterpret_cast<const uint4*>(bits + w0) + 1);
        }
        c[0] = lo.x; c[1] = lo.y; c[2] = lo.z; c[3] = lo.w;
        c[4] = hi.x; c[5] = hi.y; c[6] = hi.z; c[7] = hi.w;
#pragma unroll
        for (int i = 0; i < kRankItems; i++) {
            c[i] = __popc(c[i]);
            sum += c[i];
        }
        uint32_t incl = sum;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t t = __shfl_up_sync(kFull, incl, d);
            if (lane >= (uint32_t)d) incl += t;
        }
        if (lane == 31) s_tot[wid] = incl;
        __syncthreads();
        uint32_t t = s_tot[lane], ti = t;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t o = __shfl_up_sync(kFull, ti, d);
            if (lane >= (uint32_t)d) ti += o;
        }
        const uint32_t before = __shfl_sync(kFull, ti - t, (int)wid);
        const uint32_t all = __shfl_sync(kFull, ti, 31);
        uint32_t run = carry + before + incl - sum;
#pragma unroll
        for (int i = 0; i < kRankItems; i++) {
            const uint32_t t2 = c[i];
            c[i] = run;
            run += t2;
        }
        if (w0 < nw) {
            reinterpret_cast<uint4*>(rank + w0)[0] = make_uint4(c[0], c[1], c[2], c[3]);
            reinterpret_cast<uint4*>(rank + w0)[1] = make_uint4(c[4], c[5], c[6], c[7]);
        }
        carry += all;
        __syncthreads();
    }
    return carry;
}
// Label of the cluster that starts at visit position s.
__device__ __forceinline__ uint32_t bit_label(const uint32_t* __restrict__ bits,
                                              const uint32_t* __restrict__ rank, uint32_t s) {
    return rank[s >> 5] + __popc(bits[s >> 5] & ((1u << (s & 31u)) - 1u)) + 1u;
}

__global__ void start_flags_kernel(ClusterArgs a) {
    pdl_sync();
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= a.n || !is_core(a.deg[k], a.minpts)) return;
    if (a.parent[k] == k && a.cstart[k] == k && VDB_GUARD(a.st, a.seed[k] < a.n, 12, a.seed[k]))
        atomicOr(&a.bits[a.seed[k] >> 5], 1u << (a.seed[k] & 31u));
}

__global__ void __launch_bounds__(kRankThreads) rank_kernel(ClusterArgs a) {
    pdl_sync();
    const uint32_t k = rank_bits(a.bits, a.brank, a.nw);
    if (threadIdx.x == 0 && k) atomicAdd(&a.st->clusters, (unsigned long long)k * a.copies);
}

__device__ __forceinline__ uint32_t start_time(const ClusterArgs& a, uint32_t u) {
    return a.seed[a.cstart[a.parent[u]]];
}

// Non-core rows (shorter than minpts): earliest cluster start among the core
// neighbours that hold the point in their own neighbourhood.  (32 registers:
// the launch's 8 blocks of 256 threads per SM all stay resident.)
__global__ void __launch_bounds__(kThreads, 8) border_pull_kernel(ClusterArgs a) {
    pdl_sync();
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t r = a.row_lo + warp; r < a.row_hi; r += nwarps) {
        const uint32_t k = (uint32_t)r;
        if (is_core(a.deg[k], a.minpts)) continue;
        const unsigned long long s = a.off[k] - a.off_base, e = a.off[k + 1] - a.off_base;
        uint32_t mn = kNone;
        auto pull = [&](uint32_t v) {
            if (!VDB_GUARD(a.st, v < a.n, 11, v)) return;
            if (v == k || !is_core(a.deg[v], a.minpts)) return;
            mn = min(mn, start_time(a, v));
        };
        // one-way entries (k reaches v, v does not reach k) are skipped
        if (a.compact) {
            walk_compact_row(reinterpret_cast<const uint16_t*>(a.nbr), s, e, k, a.ptile, a.tiles,
                             a.tile_uoff, a.parts, a.trow_s, a.trow_e, 2 * a.ep->rho + 1,
                             a.unit_words, (int)lane, [&](uint32_t v, bool one_way, bool valid) {
                                 if (valid && !one_way) pull(v);
                             });
        } else {
            for (unsigned long long j = s + lane; j < e; j += 32) {
                const uint32_t ev = a.nbr[j];
                if (!(ev & kAsymFlag)) pull(ev & kIdMask);
            }
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) mn = min(mn, __shfl_down_sync(kFull, mn, d));
        if (lane == 0) a.best[k] = mn;
    }
}

// In-edges that the non-core row does not list: pairs accepted only towards
// the non-core point.
__global__ void asym_push_kernel(ClusterArgs a) {
    pdl_sync();
    uint32_t na = *a.asym_count;
    if (na > a.asym_cap) na = a.asym_cap;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < na;
         i += gridDim.x * blockDim.x) {
    const AsymPair p = a.asym[i];
    uint32_t from, to;
    if (p.dir == 1u) {
        from = p.a;
        to = p.b;
    } else {
        from = p.b;
        to = p.a;
    }
    if (!is_core(a.deg[from], a.minpts) || is_core(a.deg[to], a.minpts)) continue;
    atomicMin(&a.best[to], start_time(a, from));
    }
}

__global__ void write_labels_kernel(ClusterArgs a) {
    pdl_sync();
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= a.n) return;
    uint32_t lab;
    if (is_core(a.deg[k], a.minpts)) {
        const uint32_t t = start_time(a, k);
        lab = VDB_GUARD(a.st, t < a.n, 14, t) ? bit_label(a.bits, a.brank, t) : 0u;
    } else {
        const uint32_t b = a.best[k];
        lab = (b != kNone && b < a.gpos[k]) ? bit_label(a.bits, a.brank, b) : 0u;
    }
    if (VDB_GUARD(a.st, a.gorig[k] < a.n, 13, a.gorig[k])) a.labels_out[a.gorig[k]] = lab;
}

// ------------------------------------------------------------- cell clusters
//
// Grids whose cells are cliques (cell width <= eps/sqrt(2), 2 w^2 below the
// thresholds): the cores of a cell always share a component, so the
// union-find runs over the non-empty cells, and a border point is settled by
// its neighbour cells' cluster starts.  The neighbour table is not read.  All
// minpts of one epsilon (slots) are labelled side by side, a launch of each
// kernel for all.

// cbest[c] = largest degree of the cell (high word) and the first point that
// has it (complemented, low word): the cell has cores at minpts m iff the
// high word is >= m, and that point is one of them.
__device__ __forceinline__ uint32_t best_deg(unsigned long long b) { return (uint32_t)(b >> 32); }
__device__ __forceinline__ uint32_t best_point(unsigned long long b) { return ~(uint32_t)b; }

struct PairTest {
    bool mixed;
    float lo, hi, wf;
    ExactBounds xb;
};
__device__ __forceinline__ PairTest pair_test(const CellArgs& a) {
    PairTest t;
    t.mixed = a.ep->mixed != 0;
    t.lo = a.ep->lo32;
    t.hi = a.ep->hi32;
    t.wf = a.ep->wf;
    t.xb = a.ep->xb;
    return t;
}
// bit0: v in N(u), bit1: u in N(v), for points ku and kv whose cells lie
// (dx, dy) cells apart; pu, pv: their FP32 coordinates in their own cells.
__device__ __forceinline__ uint32_t test_pair(const CellArgs& a, const PairTest& t, uint32_t ku,
                                              uint32_t kv, float2 pu, float2 pv, int dx, int dy) {
    if (t.mixed) {
        const float ddx = __fsub_rn(pu.x, __fmaf_rn((float)dx, t.wf, pv.x));
        const float ddy = __fsub_rn(pu.y, __fadd_rn(pv.y, __fmul_rn((float)dy, t.wf)));
        const float d2 = __fmaf_rn(ddx, ddx, __fmul_rn(ddy, ddy));
        if (d2 < t.lo) return 3u;
        if (!(d2 <= t.hi)) return 0u;
    }
    return exact_pair(a.gxy[ku], a.gxy[kv], ku, kv, t.xb, a.gbox);
}

// Neighbour cells: crng[i * n + c] = the non-empty cells [x, y) of row
// i - rho within reach of cell c, ccx[c] = the column of cell c.  One thread
// per cell and row looks them up once for all slots and kernels (in sparse
// grids by binary search), so that the kernels below walk lists of cells that
// exist instead of probing every offset.
//
// The middle row's threads also set the slots' start state: no seeds, no
// cluster starts; and each cell's largest degree with its point (cbest, zero
// before).
__global__ void cell_setup_kernel(CellArgs a) {
    pdl_sync();
    if (blockIdx.y == (uint32_t)a.ep->rho) {
        const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
        if (k < a.nw)
            for (int v = 0; v < a.m; v++) a.bits[(size_t)v * a.nw + k] = 0u;
        const bool in = k < a.n;
        if (k < (uint32_t)a.m) a.st->starts_done[k] = 0u;
        if (in) {
            for (int v = 0; v < a.m; v++) a.seed[(size_t)v * a.n + k] = kNone;
        }
        const uint32_t c = in ? a.cscan[k + 1] - 1u : kNone;
        const uint32_t d = in ? a.deg[k] : 0u;
        const uint32_t same = __match_any_sync(kFull, c);
        const uint32_t mx = __reduce_max_sync(same, d);
        const uint32_t first = __reduce_min_sync(same, d == mx ? k : kNone);
        if (in && first == k && VDB_GUARD(a.st, c < a.n, 15, c))
            atomicMax(&a.cbest[c], ((unsigned long long)mx << 32) | (uint32_t)~k);
    }
    const uint32_t rho = (uint32_t)a.ep->rho;
    const uint32_t ncl = *a.ncl;
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x, r = blockIdx.y;
    if (c >= ncl || r > 2u * rho) return;
    const uint32_t key = a.gkey[a.clist[c]];
    const int cy = (int)(key / a.g.ncx_pad), cx = (int)(key - (uint32_t)cy * a.g.ncx_pad);
    const int ry = cy + (int)r - (int)rho, reach = a.ep->reach[r];
    const uint32_t lo = (uint32_t)max(cx - reach, 0);
    const uint32_t hi = (uint32_t)min(cx + reach, (int)a.g.ncx - 1);
    uint2 out = make_uint2(0u, 0u);
    if (ry >= 0 && ry < (int)a.g.ncy) {
        if (a.g.sparse) {
            const uint32_t re = a.crow[ry + 1];
            out.x = cx_lower_bound(a.ccx, a.crow[ry], re, lo);
            out.y = out.x;
            while (out.y < re && a.ccx[out.y] <= hi) out.y++;
        } else {
            const uint32_t base = (uint32_t)ry * a.g.ncx_pad;
            out.x = a.cscan[a.cell_start[base + lo]];
            out.y = a.cscan[a.cell_start[base + hi + 1]];
        }
    }
    if (!VDB_GUARD(a.st, out.x <= out.y && out.y <= ncl, 16, out.y)) out = make_uint2(0u, 0u);
    a.crng[(size_t)r * a.n + c] = out;
}

// Hooks (y: slot): at the start every cell is a tree of its own and nobody else
// writes its parent, so it can be hung under an earlier cell without atomics:
// under the first cell of the run of joined cells that it ends (within the
// warp), else under a joined cell of the row before.
//
// The slots do not build on one another.  A slot could start from the
// components of the one before (its minpts is smaller), but the hooks find most
// of them again, and the slots' kernels, each too small to fill the chip below
// 10^5 points, run as one launch (clustering of 60k points, 4 minpts of one
// epsilon, 138 -> 84 us; 2M points 564 -> 570).
__global__ void cell_hook_kernel(CellArgs a) {
    pdl_sync();
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
    const uint32_t ncl = *a.ncl;
    if (c - lane >= ncl) return;  // (whole warps)
    const bool in = c < ncl;
    const PairTest t = pair_test(a);
    const uint32_t mp = a.mp[blockIdx.y];
    const int rho = a.ep->rho;
    const unsigned long long bA = in ? a.cbest[c] : 0ull;
    const uint32_t ku = best_point(bA);
    const bool core = in && best_deg(bA) >= mp && ku < a.n;
    bool left = false;
    int cx = 0;
    float2 pu = make_float2(0.f, 0.f);
    if (core) {
        cx = (int)a.ccx[c];
        pu = a.glocal[ku];
        if (c > 0) {
            const unsigned long long bB = a.cbest[c - 1];
            const uint32_t kv = best_point(bB);
            if (best_deg(bB) >= mp && kv < a.n && (int)a.ccx[c - 1] + 1 == cx &&
                a.crng[(size_t)rho * a.n + c].x < c)  // (the same row)
                left = test_pair(a, t, ku, kv, pu, a.glocal[kv], -1, 0) == 3u;
        }
    }
    const uint32_t heads = ~__ballot_sync(kFull, left);
    uint32_t p = c;
    if (left) {
        // the run's first cell in this warp, or the cell before the warp's
        const uint32_t upto = heads & ((2u << lane) - 1u);
        p = upto ? c - lane + 31u - (uint32_t)__clz((int)upto) : c - lane - 1u;
    } else if (core && rho >= 1) {
        const uint2 rg = a.crng[(size_t)(rho - 1) * a.n + c];
        for (uint32_t o = rg.x; o < rg.y && p == c; o++) {
            const int dx = (int)a.ccx[o] - cx;
            const unsigned long long bB = a.cbest[o];
            const uint32_t kv = best_point(bB);
            if (dx >= -1 && dx <= 1 && o < c && best_deg(bB) >= mp && kv < a.n &&
                test_pair(a, t, ku, kv, pu, a.glocal[kv], dx, -1) == 3u)
                p = o;
        }
    }
    if (in) a.parent[(size_t)blockIdx.y * a.n + c] = p;
}

constexpr uint32_t kLanePairs = 4;     // cells of at most so many point pairs: one lane
constexpr uint32_t kFlatPairs = 1024;  // of at most so many: all of them, lanes over the pairs

// Unions (z: slot): every pair of cells within reach whose roots differ is
// searched for one core-core pair accepted in both directions.  A lane takes a
// cell and one row of its half neighbourhood (y; 32 cells of it at a time, a row
// has at most 5 at the default cell size): it screens the roots and tests
// the cells' points of largest degree (and all pairs of next to empty cells);
// only then the pairs that are still apart are searched by the whole warp,
// lanes over the point pairs (or, for large cells, over the first cell's points
// within eps of the second).  The searches are the expensive part, and after
// the cheap unions few are left.  The clustering of the 2M sweep at eps 0.2 took
// 0.88 ms with the cheap unions and a flatten as kernels before it, 0.67 like
// this; 1M uniform points at eps 0.05 0.50 -> 0.41 ms.
__global__ void __launch_bounds__(kThreads, 6) cell_pairs_kernel(CellArgs a) {
    pdl_sync();
    const int v = blockIdx.z;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t ncl = *a.ncl;
    const uint32_t mp = a.mp[v];
    const PairTest t = pair_test(a);
    const float near2 = a.ep->near2;
    const float wf = t.wf;
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t hrows = (uint32_t)a.ep->rho + 1u;
    const uint32_t dy = (blockIdx.y + 1u) % hrows;  // (the next row's many pairs first)
    const uint32_t skip = blockIdx.y / hrows * 32u;  // cells of the row that other blocks take
    if (c - lane >= ncl) return;  // (whole warps)
    uint32_t* parent = a.parent + (size_t)v * a.n;
    const uint32_t* __restrict__ comp = a.comp_prev[v];
    uint32_t skipped = 0;  // cell pairs of different components at a larger epsilon
    uint32_t o = 0, oe = 0, sA = 0, eA = 0, compA = kNone, ku = 0;
    int cx = 0;
    if (c < ncl) {
        const unsigned long long bA = a.cbest[c];
        ku = best_point(bA);
        if (best_deg(bA) >= mp && ku < a.n) {
            const uint2 rg = a.crng[(size_t)((uint32_t)a.ep->rho + dy) * a.n + c];
            o = (dy ? rg.x : c + 1) + skip;
            oe = min(rg.y, o + 32u);
            if (o < oe) {
                cx = (int)a.ccx[c];
                sA = a.clist[c];
                eA = a.clist[c + 1];
                if (comp) compA = comp[a.gpos[ku]];
            }
        }
    }
    // A row's cells are screened at once (their loads overlap): those with
    // cores that are not, as far as two steps up their tree show, in the cell's
    // own tree stay in `left`.
    uint32_t left = 0;
    const uint32_t o0 = o;
    {
        const uint32_t root = o < oe ? uf_find(parent, c) : 0u;
#pragma unroll 5
        for (uint32_t j = 0; j < (o < oe ? oe - o : 0u); j++) {
            if (best_deg(a.cbest[o + j]) < mp) continue;
            const uint32_t p1 = parent[o + j];
            if (p1 != root && parent[p1] != root) left |= 1u << j;
        }
    }
    // Every lane takes the cells left in its row: the cells' points of largest
    // degree first, which in dense regions mostly pair, or all points of next
    // to empty cells.  `hard` keeps the pairs that need a search.
    uint32_t hard = 0;
    while (__any_sync(kFull, left != 0u)) {
        bool join = false;
        uint32_t ra = 0, rb = 0;
        if (left) {
            const uint32_t j = (uint32_t)__ffs(left) - 1u;
            o = o0 + j;
            left &= left - 1u;
            const unsigned long long bB = a.cbest[o];
            const uint32_t kv = best_point(bB);
            ra = uf_find(parent, c);
            rb = uf_find(parent, o);
            // cores in different components at the larger epsilon are not
            // connected at this one (its components refine those)
            const bool apart = ra != rb && comp && kv < a.n && comp[a.gpos[kv]] != compA;
            if (apart) skipped++;
            if (ra != rb && !apart && kv < a.n) {
                const int dx = (int)a.ccx[o] - cx;
                join = test_pair(a, t, ku, kv, a.glocal[ku], a.glocal[kv], dx, (int)dy) == 3u;
                if (!join) {
                    const uint32_t sB = a.clist[o], eB = a.clist[o + 1];
                    if ((uint64_t)(eA - sA) * (eB - sB) <= kLanePairs) {
                        for (uint32_t u = sA; u < eA && !join; u++)
                            for (uint32_t w = sB; w < eB && !join; w++)
                                join = a.deg[u] >= mp && a.deg[w] >= mp &&
                                       test_pair(a, t, u, w, a.glocal[u], a.glocal[w], dx,
                                                 (int)dy) == 3u;
                    } else {
                        hard |= 1u << j;
                    }
                }
            }
        }
        // neighbouring lanes mostly want the same two trees joined: one union
        // per pair of roots and warp
        if (__any_sync(kFull, join)) {
            const unsigned long long key =
                join ? ((unsigned long long)max(ra, rb) << 32) | min(ra, rb) : ~0ull - lane;
            const uint32_t same = __match_any_sync(kFull, key);
            if (join && lane == (uint32_t)(__ffs(same) - 1)) uf_union(parent, ra, rb, a.st);
            __syncwarp();
        }
    }
    // the others, if their roots still differ, by the whole warp one after the
    // other
    while (__any_sync(kFull, hard != 0u)) {
        bool need = false;
        uint32_t sB = 0, eB = 0, ob = 0;
        int dx = 0;
        if (hard) {
            ob = o0 + (uint32_t)__ffs(hard) - 1u;
            hard &= hard - 1u;
            need = uf_find(parent, c) != uf_find(parent, ob);
            if (need) {
                sB = a.clist[ob];
                eB = a.clist[ob + 1];
                dx = (int)a.ccx[ob] - cx;
            }
        }
        for (uint32_t todo = __ballot_sync(kFull, need); todo; todo &= todo - 1u) {
            const int src = __ffs(todo) - 1;
            const uint32_t cA = __shfl_sync(kFull, c, src), cB = __shfl_sync(kFull, ob, src);
            // unions made since the screen may have joined the two cells
            bool joined = false;
            if (lane == 0) joined = uf_find(parent, cA) == uf_find(parent, cB);
            if (__shfl_sync(kFull, (int)joined, 0)) continue;
            const uint32_t As = __shfl_sync(kFull, sA, src), Ae = __shfl_sync(kFull, eA, src);
            const uint32_t Bs = __shfl_sync(kFull, sB, src), Be = __shfl_sync(kFull, eB, src);
            const int ox = __shfl_sync(kFull, dx, src), oy = __shfl_sync(kFull, (int)dy, src);
            const uint32_t na = Ae - As, nb = Be - Bs;
            bool found = false;
            if ((uint64_t)na * nb <= kFlatPairs) {
                const uint32_t tot = na * nb;
                for (uint32_t p0 = 0; p0 < tot && !found; p0 += 32) {
                    const uint32_t p = p0 + lane;
                    bool in = false;
                    if (p < tot) {
                        const uint32_t u = As + p / nb, w = Bs + p % nb;
                        in = a.deg[u] >= mp && a.deg[w] >= mp &&
                             test_pair(a, t, u, w, a.glocal[u], a.glocal[w], ox, oy) == 3u;
                    }
                    found = __any_sync(kFull, in);
                }
            } else {
                const float dxw = __fmul_rn((float)ox, wf), dyw = __fmul_rn((float)oy, wf);
                for (uint32_t u0 = As; u0 < Ae && !found; u0 += 32) {
                    const uint32_t u = u0 + lane;
                    bool va = u < Ae && a.deg[u] >= mp;
                    float2 pu = make_float2(0.f, 0.f);
                    if (va) {
                        // only points within eps of the other cell's square can
                        // pair (FP32 coordinates, eps^2 widened by 2^-8)
                        pu = a.glocal[u];
                        const float ex = fmaxf(fmaxf(dxw - pu.x, pu.x - (dxw + wf)), 0.0f);
                        const float ey = fmaxf(fmaxf(dyw - pu.y, pu.y - (dyw + wf)), 0.0f);
                        va = !t.mixed || __fmaf_rn(ex, ex, ey * ey) <= near2;
                    }
                    if (!__any_sync(kFull, va)) continue;
                    for (uint32_t w0 = Bs; w0 < Be && !found; w0 += 32) {
                        const uint32_t wl = w0 + lane;
                        bool vb = wl < Be && a.deg[wl] >= mp;
                        float2 pw = make_float2(0.f, 0.f);
                        if (vb) {
                            pw = a.glocal[wl];
                            const float bx = __fmaf_rn((float)ox, wf, pw.x);
                            const float by = __fadd_rn(pw.y, dyw);
                            const float ex = fmaxf(fmaxf(-bx, bx - wf), 0.0f);
                            const float ey = fmaxf(fmaxf(-by, by - wf), 0.0f);
                            vb = !t.mixed || __fmaf_rn(ex, ex, ey * ey) <= near2;
                        }
                        for (uint32_t cm = __ballot_sync(kFull, vb); cm && !found; cm &= cm - 1u) {
                            const int s1 = __ffs(cm) - 1;
                            const float2 q = make_float2(__shfl_sync(kFull, pw.x, s1),
                                                         __shfl_sync(kFull, pw.y, s1));
                            const bool in = va && test_pair(a, t, u, w0 + (uint32_t)s1, pu, q, ox,
                                                            oy) == 3u;
                            found = __any_sync(kFull, in);
                        }
                    }
                }
            }
            if (found && lane == 0) uf_union(parent, cA, cB, a.st);
            __syncwarp();
        }
    }
    skipped = __reduce_add_sync(kFull, skipped);
    if (lane == 0 && skipped) atomicAdd(&a.st->reuse_skips, (unsigned long long)skipped);
}

// Roots, and seed[root] = first visit position among the component's cores (y:
// slot).  Each core walks up its cell's tree, in a few steps that its
// neighbours in cell order share; the cell's first point leaves the root.
__global__ void cell_seed_kernel(CellArgs a) {
    pdl_sync();
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    const int v = blockIdx.y;
    if (k >= a.n) return;
    const bool core = a.deg[k] >= a.mp[v];
    const uint32_t before = a.cscan[k], c = a.cscan[k + 1] - 1u;
    const bool first = before == c;  // of its cell
    if (!core && !first) return;
    if (!VDB_GUARD(a.st, c < a.n, 16, c)) return;
    uint32_t* parent = a.parent + (size_t)v * a.n;
    const uint32_t r = uf_find_ro(parent, c);
    if (first) parent[c] = r;
    if (!core) return;
    // neighbours in cell order mostly share a root: one atomic per root and warp
    const uint32_t same = __match_any_sync(__activemask(), r);
    const uint32_t mn = __reduce_min_sync(same, a.gpos[k]);
    if ((threadIdx.x & 31) == (uint32_t)(__ffs(same) - 1) && r < a.n)
        atomicMin(&a.seed[(size_t)v * a.n + r], mn);
}

// Core-core edges accepted in one direction only, between components (one
// thread per slot; run only when the table has one-way pairs): the components
// that an earlier cluster's expansion absorbs take its start as their seed.
__global__ void cell_resolve_kernel(CellArgs a, uint32_t* ws, uint32_t cap) {
    pdl_sync();
    if (threadIdx.x != 0) return;
    const int v = blockIdx.x;
    const uint32_t mp = a.mp[v];
    const uint32_t* parent = a.parent + (size_t)v * a.n;
    uint32_t* seed = a.seed + (size_t)v * a.n;
    uint32_t* cs = a.cst + (size_t)v * a.n;  // start component of the edges' components
    ws += (size_t)v * 6 * cap;
    uint32_t na = *a.asym_count;
    if (na > a.asym_cap) na = a.asym_cap;
    uint32_t* efrom = ws;
    uint32_t* eto = ws + cap;
    uint32_t* nodes = ws + 2 * cap;
    uint32_t* stack = ws + 4 * cap;  // 2*cap entries
    uint32_t ne = 0;
    for (uint32_t i = 0; i < na; i++) {
        const AsymPair p = a.asym[i];
        if (a.deg[p.a] < mp || a.deg[p.b] < mp) continue;
        const uint32_t ra = parent[a.cscan[p.a + 1] - 1u], rb = parent[a.cscan[p.b + 1] - 1u];
        if (ra == rb) continue;
        if (ne >= cap) {
            atomicOr(&a.st->flags, kStatResolveOverflow);
            return;
        }
        // dir 1: b in N(a) only, a's expansion reaches b
        efrom[ne] = p.dir == 1u ? ra : rb;
        eto[ne] = p.dir == 1u ? rb : ra;
        ne++;
    }
    if (ne == 0) return;
    // distinct endpoint components in seed order
    uint32_t nn = 0;
    for (uint32_t i = 0; i < 2 * ne; i++) {
        const uint32_t r = i < ne ? efrom[i] : eto[i - ne];
        bool dup = false;
        for (uint32_t j = 0; j < nn && !dup; j++) dup = nodes[j] == r;
        if (dup) continue;
        uint32_t j = nn++;
        while (j > 0 && seed[nodes[j - 1]] > seed[r]) {
            nodes[j] = nodes[j - 1];
            j--;
        }
        nodes[j] = r;
    }
    for (uint32_t i = 0; i < nn; i++) cs[nodes[i]] = kNone;
    for (uint32_t i = 0; i < nn; i++) {
        const uint32_t u = nodes[i];
        if (cs[u] != kNone) continue;
        cs[u] = u;
        uint32_t top = 0;
        stack[top++] = u;
        while (top) {
            const uint32_t x = stack[--top];
            for (uint32_t e = 0; e < ne; e++) {
                if (efrom[e] != x) continue;
                const uint32_t y = eto[e];
                if (cs[y] != kNone) continue;
                cs[y] = u;
                stack[top++] = y;
            }
        }
    }
    for (uint32_t i = 0; i < nn; i++) seed[nodes[i]] = seed[cs[nodes[i]]];
}

// cst = visit position at which the cluster of the cell's cores starts (kNone:
// no cores); the starts' bits (y: slot).  The slot's last block ranks the bits
// and counts the clusters.
__global__ void __launch_bounds__(kRankThreads) cell_starts_kernel(CellArgs a) {
    pdl_sync();
    __shared__ bool s_last;
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    const int v = blockIdx.y;
    uint32_t* const bits = a.bits + (size_t)v * a.nw;
    if (c < *a.ncl) {
        const size_t o = (size_t)v * a.n;
        uint32_t s = kNone;
        if (best_deg(a.cbest[c]) >= a.mp[v]) {
            const uint32_t r = a.parent[o + c];
            s = r < a.n ? a.seed[o + r] : kNone;
            if (!VDB_GUARD(a.st, s < a.n, 12, s)) s = kNone;
            else if (r == c) atomicOr(&bits[s >> 5], 1u << (s & 31u));
        }
        a.cst[o + c] = s;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(&a.st->starts_done[v], 1u) == gridDim.x - 1u;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const uint32_t k = rank_bits(bits, a.brank + (size_t)v * a.nw, a.nw);
    if (threadIdx.x == 0 && k) atomicAdd(&a.st->clusters, (unsigned long long)k * a.copies[v]);
}

// Label of the cluster that starts at visit position s.
__device__ __forceinline__ uint32_t start_label(const CellArgs& a, int v, uint32_t s) {
    return bit_label(a.bits + (size_t)v * a.nw, a.brank + (size_t)v * a.nw, s);
}

// Labels, a thread per point and slot (y), and the saved components
// (comp[visit position] = cluster start of the core there, kNone for other
// points).  A core has its cell's cluster.  A point p that is not core
// takes the earliest cluster start among the cores u with p in N(u): the
// start of its own cell if that has cores (a clique), or of a neighbour cell
// if one of that cell's cores lists p.  Only neighbour cells whose start is
// earlier than what p has are searched, earliest start first: a point whose
// neighbour cells all belong to its own cell's cluster searches nothing, and
// one surrounded by a single other cluster ends at the first core found.  A
// start after p's own visit position cannot label it (p was visited first, as
// noise).  The lanes of a warp search side by side while there are at most
// kLaneCores points for each lane that searches; a few lanes' larger searches
// are done by the warp one after the other, lanes over the cells' points (a lane
// holds a row, so not on grids of more than 32 rows, 16 and more cells per
// epsilon).
constexpr uint32_t kLaneCores = 16;
__global__ void __launch_bounds__(kThreads, 8) cell_labels_kernel(CellArgs a) {
    pdl_sync();
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    const int v = blockIdx.y;
    const uint32_t mp = a.mp[v];
    const uint32_t* __restrict__ cst = a.cst + (size_t)v * a.n;
    uint32_t c = 0, p = 0, out = 0, best = 0;
    bool border = false;
    if (k < a.n) {
        const uint32_t d = a.deg[k];
        c = a.cscan[k + 1] - 1u;
        p = a.gpos[k];
        out = a.gorig[k];
        if (VDB_GUARD(a.st, c < a.n && out < a.n && p < a.n, 13, out)) {
            best = cst[c];
            border = d < mp;
            if (!border) {
                if (VDB_GUARD(a.st, best < a.n, 14, best)) a.labels[v][out] = start_label(a, v, best);
            }
            if (a.comp_out[v]) a.comp_out[v][p] = border ? kNone : best;
        }
    }
    if (!__any_sync(kFull, border)) return;
    const PairTest t = pair_test(a);
    const int rho = a.ep->rho, nrows = 2 * rho + 1;
    int cx = 0;
    float2 loc = make_float2(0.f, 0.f);
    if (border) {
        cx = (int)a.ccx[c];
        loc = a.glocal[k];
    }
    const uint2* __restrict__ rng = a.crng + c;  // row i: rng[i * n]
    {
        uint32_t floor_s = 0;  // starts below this one have been searched
        bool busy = border;
        while (__any_sync(kFull, busy)) {
            // the earliest start that is left among the neighbour cells
            uint32_t ms = kNone;
            if (busy) {
                const uint32_t lim = min(best, p);
                for (int i = 0; i < nrows; i++) {
                    const uint2 rg = rng[(size_t)i * a.n];
                    const uint32_t cnt = rg.y - rg.x;
#pragma unroll 2
                    for (uint32_t j = 0; j < cnt; j++) {
                        const uint32_t st = cst[rg.x + j];
                        ms = min(ms, st >= floor_s ? st : kNone);
                    }
                }
                if (ms >= lim) {
                    ms = kNone;
                    busy = false;
                }
            }
            if (!__any_sync(kFull, busy)) break;
            // the points of its cells
            uint32_t npts = 0;
            if (busy) {
                for (int i = 0; i < nrows; i++) {
                    const uint2 rg = rng[(size_t)i * a.n];
                    for (uint32_t o = rg.x; o < rg.y; o++)
                        if (cst[o] == ms) npts += a.clist[o + 1] - a.clist[o];
                }
            }
            bool hit = false;
            const uint32_t searching = (uint32_t)__popc(__ballot_sync(kFull, busy));
            const bool wide = busy && nrows <= 32 && npts > kLaneCores * searching;
            if (busy && !wide) {
                for (int j = 0; j < nrows && !hit; j++) {
                    const int dy = (j + 1) / 2 * ((j & 1) ? 1 : -1);  // nearest rows first
                    const uint2 rg = rng[(size_t)(dy + rho) * a.n];
                    for (uint32_t o = rg.x; o < rg.y && !hit; o++) {
                        if (cst[o] != ms) continue;
                        const int dx = (int)a.ccx[o] - cx;
                        const uint32_t e = a.clist[o + 1];
                        for (uint32_t u = a.clist[o]; u < e && !hit; u++)
                            hit = a.deg[u] >= mp &&
                                  (test_pair(a, t, k, u, loc, a.glocal[u], dx, dy) & 2u);
                    }
                }
            }
            for (uint32_t todo = __ballot_sync(kFull, wide); todo; todo &= todo - 1u) {
                const int src = __ffs(todo) - 1;
                const uint32_t kk = __shfl_sync(kFull, k, src), cc = __shfl_sync(kFull, c, src);
                const uint32_t mss = __shfl_sync(kFull, ms, src);
                const int cxx = __shfl_sync(kFull, cx, src);
                const float2 l = make_float2(__shfl_sync(kFull, loc.x, src),
                                             __shfl_sync(kFull, loc.y, src));
                // lanes over the rows' ranges, then over the cells: the cells
                // with that start, each with its points
                uint2 rg = make_uint2(0u, 0u);
                if ((int)lane < nrows) rg = a.crng[(size_t)lane * a.n + cc];
                uint32_t incl = rg.y - rg.x;
#pragma unroll
                for (int s1 = 1; s1 < 32; s1 <<= 1) {
                    const uint32_t x = __shfl_up_sync(kFull, incl, s1);
                    if ((int)lane >= s1) incl += x;
                }
                const uint32_t ncells = __shfl_sync(kFull, incl, 31);
                bool found = false;
                for (uint32_t base = 0; base < ncells && !found; base += 32) {
                    const uint32_t j = base + lane;
                    uint32_t o = 0;
                    int row = 0;
                    for (int i = 0; i < nrows; i++) {
                        const uint32_t ie = __shfl_sync(kFull, incl, i);
                        const uint2 rr = make_uint2(__shfl_sync(kFull, rg.x, i),
                                                    __shfl_sync(kFull, rg.y, i));
                        if (j < ie && j >= ie - (rr.y - rr.x)) {
                            o = rr.x + (j - (ie - (rr.y - rr.x)));
                            row = i;
                        }
                    }
                    const bool mine = j < ncells && cst[o] == mss;
                    uint32_t b = 0, e = 0;
                    int dx = 0;
                    if (mine) {
                        b = a.clist[o];
                        e = a.clist[o + 1];
                        dx = (int)a.ccx[o] - cxx;
                    }
                    // nearest cells first
                    const int gx = max(abs(dx) - 1, 0), gy = max(abs(row - rho) - 1, 0);
                    uint32_t left = __ballot_sync(kFull, mine);
                    const uint32_t order = ((uint32_t)(gx * gx + gy * gy) << 5) | lane;
                    while (left && !found) {
                        const uint32_t pick =
                            __reduce_min_sync(kFull, (left >> lane) & 1u ? order : kNone) & 31u;
                        left &= ~(1u << pick);
                        const uint32_t bb = __shfl_sync(kFull, b, (int)pick);
                        const uint32_t ee = __shfl_sync(kFull, e, (int)pick);
                        const int ox = __shfl_sync(kFull, dx, (int)pick);
                        const int oy = __shfl_sync(kFull, row, (int)pick) - rho;
                        for (uint32_t u0 = bb; u0 < ee && !found; u0 += 32) {
                            const uint32_t u = u0 + lane;
                            const bool in = u < ee && a.deg[u] >= mp &&
                                            (test_pair(a, t, kk, u, l, a.glocal[u], ox, oy) & 2u);
                            found = __any_sync(kFull, in);
                        }
                    }
                }
                if (found && (int)lane == src) hit = true;
            }
            if (busy) {
                if (hit) {
                    best = ms;
                    busy = false;  // (no earlier start is left)
                } else {
                    floor_s = ms + 1u;
                }
            }
        }
        if (border) a.labels[v][out] = best < p ? start_label(a, v, best) : 0u;
    }
}

}  // namespace

size_t resolve_scratch_bytes() { return (size_t)kResolveCap * 6 * sizeof(uint32_t); }

void launch_uf_init(const ClusterArgs& a, bool fresh, cudaStream_t s) {
    if (!a.n) return;
    launch(uf_init_kernel, nblk(std::max(a.n, a.nw)), kThreads, s, a, fresh ? 1 : 0);
}

void launch_uf_union(const ClusterArgs& a, int nblocks, cudaStream_t s) {
    if (a.row_hi > a.row_lo) { launch(uf_union_kernel, nblocks, kThreads, s, a); }
}

void launch_uf_finish(const ClusterArgs& a, void* resolve_ws, cudaStream_t s) {
    if (!a.n) return;
    launch(uf_flatten_kernel, nblk(a.n), kThreads, s, a);
    launch(resolve_kernel, 1, 32, s, a, (uint32_t*)resolve_ws, kResolveCap);
    launch(start_flags_kernel, nblk(a.n), kThreads, s, a);
    launch(rank_kernel, 1, kRankThreads, s, a);
}

void launch_save_components(const ClusterArgs& a, uint32_t* comp, cudaStream_t s) {
    if (!a.n) return;
    launch(save_components_kernel, nblk(a.n), kThreads, s, a, comp);
}

void launch_border_pull(const ClusterArgs& a, int nblocks, cudaStream_t s) {
    if (a.row_hi <= a.row_lo) return;
    launch(border_pull_kernel, nblocks, kThreads, s, a);
}

void launch_label_write(const ClusterArgs& a, cudaStream_t s) {
    if (!a.n) return;
    launch(asym_push_kernel, 64, kThreads, s, a);
    launch(write_labels_kernel, nblk(a.n), kThreads, s, a);
}

void launch_border_and_write(const ClusterArgs& a, int nblocks, cudaStream_t s) {
    if (!a.n) return;
    launch_border_pull(a, nblocks, s);
    launch_label_write(a, s);
}

void launch_cells(const CellArgs& a, int nrows, int row_cells, bool one_way, void* resolve_ws,
                  cudaStream_t s) {
    if (!a.n) return;
    const unsigned parts = (unsigned)(row_cells + 31) / 32u;
    const dim3 per_slot(nblk(a.n), (unsigned)a.m);
    launch(cell_setup_kernel, dim3(nblk(std::max(a.n, a.nw)), (unsigned)nrows), kThreads, s, a);
    launch(cell_hook_kernel, per_slot, kThreads, s, a);
    launch(cell_pairs_kernel, dim3(nblk(a.n), (unsigned)(nrows / 2 + 1) * parts, (unsigned)a.m),
           kThreads, s, a);
    launch(cell_seed_kernel, per_slot, kThreads, s, a);
    if (one_way) {
        launch(cell_resolve_kernel, a.m, 32, s, a, (uint32_t*)resolve_ws, kResolveCap);
    }
    launch(cell_starts_kernel, dim3((a.n + kRankThreads - 1) / kRankThreads, (unsigned)a.m),
           kRankThreads, s, a);
    launch(cell_labels_kernel, per_slot, kThreads, s, a);
}

}  // namespace vdb
