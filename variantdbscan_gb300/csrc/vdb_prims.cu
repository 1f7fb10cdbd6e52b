// Device primitives: single-pass scans, a stable LSD radix sort of (key, value)
// pairs and the dataset bounding-box reduction.
#include <float.h>

#include "vdb_lookback.cuh"

namespace vdb {

std::atomic<unsigned long long> g_launches{0};
thread_local bool g_plain_launch = false;

// ------------------------------------------------------------------ scan
//
// One kernel: blocks take their tiles in order (a ticket), publish the tile's
// sum and look back over the tiles before it (block_lookback), so the input is
// read once and a scan is one launch.  With three kernels per scan the small
// datasets' calls spent a third of their launches on scans.

namespace {

constexpr int kScanItems = 8;
constexpr uint32_t kScanTile = kLookThreads * kScanItems;

__global__ void __launch_bounds__(kLookThreads) scan_kernel(const uint32_t* __restrict__ in,
                                                            unsigned long long* __restrict__ out,
                                                            uint32_t n, LookState ls,
                                                            DeviceStatus* st) {
    pdl_sync();
    const uint32_t tile = lookback_ticket(ls);
    const uint64_t base = (uint64_t)tile * kScanTile + threadIdx.x * kScanItems;
    uint32_t v[kScanItems];
    unsigned long long sum = 0;
    if (base + kScanItems <= n) {
        const uint4 a = *reinterpret_cast<const uint4*>(in + base);
        const uint4 b = *reinterpret_cast<const uint4*>(in + base + 4);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
        v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
#pragma unroll
        for (int i = 0; i < kScanItems; i++) v[i] = base + i < n ? in[base + i] : 0u;
    }
#pragma unroll
    for (int i = 0; i < kScanItems; i++) sum += v[i];
    unsigned long long run = block_lookback(sum, tile, ls, st);
    if (base + kScanItems < n) {
        // (out is 16-byte aligned: whole sectors at a time)
#pragma unroll
        for (int i = 0; i < kScanItems; i += 2) {
            reinterpret_cast<ulonglong2*>(out + base)[i / 2] = make_ulonglong2(run, run + v[i]);
            run += (unsigned long long)v[i] + v[i + 1];
        }
        return;
    }
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        if (base + i < n) out[base + i] = run;
        run += v[i];
        if (base + i + 1 == n) {
            out[n] = run;
            st->entries = run;
        }
    }
}

}  // namespace

size_t scan_state_bytes(uint32_t n) { return look_state_bytes((n + kScanTile - 1) / kScanTile); }

void scan_u32_to_u64(const uint32_t* in, unsigned long long* out, uint32_t n, void* state,
                     DeviceStatus* st, cudaStream_t s) {
    if (!n) return;
    const uint32_t nb = (n + kScanTile - 1) / kScanTile;
    launch(scan_kernel, nb, kLookThreads, s, in, out, n, look_state(state), st);
}

// ------------------------------------------------------------------ radix sort
//
// A one-sweep sort (Adinets and Merrill 2022) with digits of 9 bits (27-bit keys
// take three passes, the 17 bits of the visit order two).  The kernel that makes
// the keys also counts all their digits, so a pass is one kernel: a block ranks
// its tile's keys per digit, looks back over the tiles before it, a thread per
// digit, and writes every pair to its place.  Pairs travel as 8 bytes between passes; the last
// pass writes the two arrays.  Measured on 1M keys of 25 bits: 3 launches and
// 85 us against 20 launches and 140 us with separate histogram and scan
// kernels per 8-bit digit.

namespace {

constexpr int kSortWarps = kDigits / 32;  // a thread per digit

template <int ITEMS>
__global__ void __launch_bounds__(kDigits) radix_pass_kernel(
    const uint32_t* __restrict__ keys_in, const uint2* __restrict__ in, uint2* __restrict__ out,
    uint32_t* __restrict__ okeys, uint32_t* __restrict__ ovals, uint32_t* __restrict__ oinv,
    uint32_t n, int shift, int drop, const uint32_t* __restrict__ hist,
    unsigned long long* __restrict__ state, uint32_t* __restrict__ ticket, DeviceStatus* st) {
    pdl_sync();
    __shared__ uint16_t s_cnt[kSortWarps][kDigits];
    __shared__ uint32_t s_base[kDigits];
    __shared__ uint32_t s_warp[kSortWarps];
    __shared__ uint32_t s_tile;
    const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    for (uint32_t i = tid; i < kSortWarps * kDigits / 2; i += kDigits)
        reinterpret_cast<uint32_t*>(s_cnt)[i] = 0u;
    if (tid == 0) s_tile = atomicAdd(ticket, 1u);
    // first place of every digit: exclusive scan of the histogram
    const uint32_t h = hist[tid];
    uint32_t incl = h;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= (uint32_t)d) incl += v;
    }
    if (lane == 31) s_warp[wid] = incl;
    __syncthreads();
    uint32_t gbase = incl - h;
    for (uint32_t w = 0; w < wid; w++) gbase += s_warp[w];
    const uint32_t tile = s_tile;
    // a warp takes 32 * ITEMS consecutive keys; item i of lane l is number 32 i + l
    const uint64_t seg = (uint64_t)tile * (kDigits * ITEMS) + wid * (32u * ITEMS);
    uint32_t key[ITEMS], val[ITEMS], rank[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
        const uint64_t k = seg + 32u * i + lane;
        key[i] = val[i] = 0;
        if (k < n) {
            if (keys_in) {
                key[i] = keys_in[k];
                val[i] = (uint32_t)k;
            } else {
                const uint2 p = in[k];
                key[i] = p.x;
                val[i] = p.y;
            }
        }
    }
    const uint32_t lt = (1u << lane) - 1u;
    uint16_t* cnt = s_cnt[wid];
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
        const bool valid = seg + 32u * i + lane < n;
        const uint32_t d = valid ? (key[i] >> shift) & (kDigits - 1u) : kDigits + lane;
        const uint32_t peers = __match_any_sync(0xffffffffu, d);
        uint32_t b = 0;
        if (valid) b = cnt[d];
        __syncwarp();
        if (valid && (peers & lt) == 0u) cnt[d] = (uint16_t)(b + __popc(peers));
        __syncwarp();
        rank[i] = b + __popc(peers & lt);
    }
    __syncthreads();
    // thread = digit: the warps' counts become offsets within the tile
    uint32_t total = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; w++) {
        const uint32_t c = s_cnt[w][tid];
        s_cnt[w][tid] = (uint16_t)total;
        total += c;
    }
    s_base[tid] = gbase + (uint32_t)digit_lookback(total, tile, state + tid, kDigits, st);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
        if (seg + 32u * i + lane >= n) continue;
        const uint32_t d = (key[i] >> shift) & (kDigits - 1u);
        const uint32_t dst = s_base[d] + cnt[d] + rank[i];
        if (dst >= n) continue;  // (only after a failed look-back, which is reported)
        if (out) {
            out[dst] = make_uint2(key[i], val[i]);
        } else {
            if (okeys) okeys[dst] = key[i] >> drop;
            ovals[dst] = val[i];
            if (oinv) oinv[val[i]] = dst;
        }
    }
}

// Keys per thread: short tiles for small sorts, so that they spread over the
// chip (50k keys: 49 tiles of 1,024 instead of 13 of 4,096), long ones where
// they still fill it.  Index of one epsilon (five passes), us, with 2 / 4 / 8 / 16
// keys: 130k points 123 / 124 / 127 / 150, 262k 160 / 158 / 162 / 171, 524k 199 / 188
// / 207 / 201, 800k 253 / 232 / 236 / 226, 1M 294 / 269 / 259 / 246.
int sort_items(uint32_t n) { return n <= (1u << 18) ? 2 : n <= (3u << 18) ? 4 : 16; }

template <int ITEMS>
void run_pass(uint32_t nb, const uint32_t* keys_in, const uint2* in, uint2* out, uint32_t* okeys,
              uint32_t* ovals, uint32_t* oinv, uint32_t n, int shift, int drop,
              const uint32_t* hist, unsigned long long* state, uint32_t* ticket, DeviceStatus* st,
              cudaStream_t s) {
    launch(radix_pass_kernel<ITEMS>, nb, kDigits, s, keys_in, in, out, okeys, ovals, oinv, n, shift,
                                                    drop, hist, state, ticket, st);
}

uint32_t sort_blocks(uint32_t n) {
    const uint32_t tile = (uint32_t)(kDigits * sort_items(n));
    return (uint32_t)(((uint64_t)n + tile - 1) / tile);
}

}  // namespace

// (keys of no bits are all equal: one pass puts every pair in its place)
int sort_passes(int bits) { return std::max(1, (bits + kDigitBits - 1) / kDigitBits); }

// zeroed memory of a sort: digit counts, tickets, look-back states
size_t sort_zero_bytes(uint32_t n, int bits) {
    const size_t p = (size_t)sort_passes(bits);
    return p * kDigits * 4 + 256 + p * (size_t)sort_blocks(n) * kDigits * 8;
}
size_t sort_scratch_bytes(uint32_t n) { return (size_t)n * 16; }

void radix_sort(const uint32_t* keys, uint32_t n, int bits, int drop, void* zeroed, void* scratch,
                uint32_t* okeys, uint32_t* ovals, uint32_t* oinv, DeviceStatus* st,
                cudaStream_t s) {
    if (!n) return;
    const int p = sort_passes(bits);
    const uint32_t nb = sort_blocks(n);
    uint32_t* hist = (uint32_t*)zeroed;
    uint32_t* ticket = hist + (size_t)p * kDigits;
    unsigned long long* state = (unsigned long long*)((char*)zeroed + (size_t)p * kDigits * 4 + 256);
    uint2* buf[2] = {(uint2*)scratch, (uint2*)scratch + n};
    const int items = sort_items(n);
    for (int i = 0; i < p; i++) {
        const bool last = i == p - 1;
        const uint32_t* kin = i == 0 ? keys : nullptr;
        const uint2* in = i == 0 ? nullptr : buf[(i - 1) & 1];
        uint2* out = last ? nullptr : buf[i & 1];
        auto pass = items == 2 ? run_pass<2> : items == 4 ? run_pass<4> : run_pass<16>;
        pass(nb, kin, in, out, last ? okeys : nullptr, last ? ovals : nullptr, last ? oinv : nullptr,
             n, i * kDigitBits, last ? drop : 0, hist + (size_t)i * kDigits,
             state + (size_t)i * nb * kDigits, ticket + i, st, s);
    }
}

// ------------------------------------------------------------------ bounding box

namespace {

constexpr int kBoxThreads = 256;

// The box's four sides, each as a maximum: ~key(min x), key(max x), ~key(min y),
// key(max y) of the ordered keys.
struct BoxAcc {
    unsigned long long m[4];
};

__device__ __forceinline__ void box_merge(BoxAcc& a, const BoxAcc& b) {
#pragma unroll
    for (int i = 0; i < 4; i++) a.m[i] = max(a.m[i], b.m[i]);
}

// The block's box: side l in lane l (of 4) of its first warp.
__device__ __forceinline__ unsigned long long box_block_reduce(const BoxAcc& v) {
    static_assert(kBoxThreads == 256, "eight warps, four sides: one lane each");
    __shared__ unsigned long long sh[kBoxThreads / 32][4];
    const uint32_t lane = threadIdx.x & 31;
    unsigned long long mine = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const unsigned long long r = warp_max_u64(v.m[i]);
        if ((int)lane == i) mine = r;
    }
    __syncthreads();  // (a call before this one has read the shared words)
    if (lane < 4) sh[threadIdx.x >> 5][lane] = mine;
    __syncthreads();
    unsigned long long r = 0;
    if (threadIdx.x < 32) {
        r = sh[lane >> 2][lane & 3];
#pragma unroll
        for (int d = 4; d < 32; d <<= 1) r = max(r, __shfl_xor_sync(0xffffffffu, r, d));
    }
    return r;
}

// The block that finishes last merges the parts.  done (zero at the launch)
// counts the blocks, and in its upper half those with a value that is not
// finite (such values stay out of the box).  With FP64 minima the FP64 pipe was
// the bound: 12.5 us for 50k points and 29 for 1M.
__global__ void __launch_bounds__(kBoxThreads) bbox_kernel(const double* __restrict__ x,
                                                           const double* __restrict__ y,
                                                           uint32_t n, BoxAcc* part,
                                                           uint32_t* done, BBox* out) {
    pdl_sync();
    __shared__ uint32_t s_done;
    const unsigned long long kmax = ordered_key(DBL_MAX), kmin = ordered_key(-DBL_MAX);
    const BoxAcc none{{~kmax, kmin, ~kmax, kmin}};
    BoxAcc a = none;
    bool bad = false;
#pragma unroll 4
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const double xi = x[i], yi = y[i];
        const unsigned long long kx = ordered_key(xi), ky = ordered_key(yi);
        const bool fx = kx >= kmin && kx <= kmax, fy = ky >= kmin && ky <= kmax;
        bad |= !fx || !fy;
        box_merge(a, BoxAcc{{fx ? ~kx : 0ull, fx ? kx : 0ull, fy ? ~ky : 0ull, fy ? ky : 0ull}});
    }
    const unsigned long long r = box_block_reduce(a);
    bad = __syncthreads_or(bad);
    if (threadIdx.x < 32) {
        if (threadIdx.x < 4) {
            part[blockIdx.x].m[threadIdx.x] = r;
            __threadfence();
        }
        __syncwarp();
        if (threadIdx.x == 0) {
            const uint32_t add = bad ? 0x10001u : 1u;
            s_done = atomicAdd(done, add) + add;
        }
    }
    __syncthreads();
    const uint32_t counts = s_done;
    if ((counts & 0xffffu) != gridDim.x) return;
    __threadfence();
    a = none;
    for (uint32_t i = threadIdx.x; i < gridDim.x; i += blockDim.x) {
        const volatile BoxAcc* p = part + i;
        box_merge(a, BoxAcc{{p->m[0], p->m[1], p->m[2], p->m[3]}});
    }
    unsigned long long s = box_block_reduce(a);
    if (threadIdx.x < 4) {
        if (!(threadIdx.x & 1)) s = ~s;
        const double v = ordered_value(s);
        // src/main.cpp:465-488: min starts at DBL_MAX, max at DBL_MIN
        if (threadIdx.x == 0) out->minx = v;
        if (threadIdx.x == 2) out->miny = v;
        if (threadIdx.x == 1) {
            out->maxx = fmax(v, DBL_MIN);
            out->tmaxx = v;
        }
        if (threadIdx.x == 3) {
            out->maxy = fmax(v, DBL_MIN);
            out->tmaxy = v;
            out->nonfinite = counts >> 16 ? 1u : 0u;
            out->pad = 0;
        }
    }
}

constexpr int kBoxBlocks = 608;  // four per SM (and below 2^16: see done)

}  // namespace

size_t bbox_scratch_bytes() { return sizeof(BoxAcc) * kBoxBlocks; }

void launch_bbox(const double* x, const double* y, uint32_t n, BBox* out, void* scratch,
                 uint32_t* zeroed, cudaStream_t s) {
    const int nb = (int)std::max<uint32_t>(1u, std::min<uint32_t>(kBoxBlocks, (n + 511u) / 512u));
    launch(bbox_kernel, nb, kBoxThreads, s, x, y, n, (BoxAcc*)scratch, zeroed, out);
}

}  // namespace vdb
