// Single-pass prefix sums (decoupled look-back, Merrill and Garland 2016): a
// tile publishes its own sum, then adds up what the tiles before it have
// published, back to the first that knows its whole prefix.  Tiles are taken
// by ticket, so every tile before a running one has started.  A state is one
// 64-bit word (two flag bits, 62 bits of sum), so a plain load sees both.
// States and tickets are zero at the launch.
#pragma once

#include <algorithm>

#include "vdb_internal.cuh"

namespace vdb {

constexpr int kLookThreads = 256;
constexpr unsigned long long kLookSum = 1ull << 62;     // the tile's own sum
constexpr unsigned long long kLookPrefix = 2ull << 62;  // the sum of all tiles up to this one
constexpr unsigned long long kLookMask = (1ull << 62) - 1ull;
// Polls of one state before the wait is given up (and reported as a failed
// index guard): far above what a running tile takes to publish.
constexpr int kLookPolls = 1 << 22;
constexpr uint32_t kLookSite = 20;

struct LookState {
    uint32_t* ticket;
    unsigned long long* tiles;
};
inline size_t look_state_bytes(uint64_t ntiles) { return 16 + (size_t)ntiles * 8; }
inline LookState look_state(void* zeroed) {
    return LookState{(uint32_t*)zeroed, (unsigned long long*)((char*)zeroed + 16)};
}

static __device__ __forceinline__ unsigned long long look_load(const unsigned long long* p) {
    return *(const volatile unsigned long long*)p;
}
static __device__ __forceinline__ void look_store(unsigned long long* p, unsigned long long v) {
    *(volatile unsigned long long*)p = v;
}
// A published state of *p (waits for it).
static __device__ __forceinline__ unsigned long long look_wait(const unsigned long long* p,
                                                               DeviceStatus* st) {
    unsigned long long v = look_load(p);
    for (int i = 0; (v >> 62) == 0ull && i < kLookPolls; i++) v = look_load(p);
    if ((v >> 62) == 0ull) {
        guard_fail(st, kLookSite, 0);
        v = kLookPrefix;
    }
    return v;
}

// The block's tile (every thread).
static __device__ __forceinline__ uint32_t lookback_ticket(LookState ls) {
    __shared__ uint32_t s_ticket;
    if (threadIdx.x == 0) s_ticket = atomicAdd(ls.ticket, 1u);
    __syncthreads();
    return s_ticket;
}

// One warp: what the tiles before this one add up to (every lane), all being
// this tile's own sum; 32 tiles are looked at at a time.
static __device__ __forceinline__ unsigned long long warp_lookback(unsigned long long all,
                                                                   uint32_t tile,
                                                                   unsigned long long* tiles,
                                                                   DeviceStatus* st) {
    const uint32_t lane = threadIdx.x & 31;
    unsigned long long before = 0;
    if (tile == 0) {
        if (lane == 0) look_store(&tiles[0], kLookPrefix | all);
        return 0;
    }
    if (lane == 0) look_store(&tiles[tile], kLookSum | all);
    for (int64_t b = (int64_t)tile - 1; b >= 0; b -= 32) {
        const int64_t i = b - (int64_t)lane;
        const unsigned long long s = i >= 0 ? look_wait(&tiles[i], st) : kLookPrefix;
        const uint32_t full = __ballot_sync(0xffffffffu, (s >> 62) == 2ull);
        const uint32_t upto = full ? (uint32_t)__ffs(full) - 1u : 31u;
        unsigned long long add = lane <= upto ? s & kLookMask : 0ull;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) add += __shfl_xor_sync(0xffffffffu, add, d);
        before += add;
        if (full) break;
    }
    if (lane == 0) look_store(&tiles[tile], kLookPrefix | (before + all));
    return before;
}

// Exclusive prefixes of this thread's K values v[] over all tiles' threads, in
// place (blocks of kLookThreads).  Warp i looks back for value i, so that
// several sums wait side by side.  (Once per kernel: the shared words are not
// guarded against a second call.)
template <int K>
static __device__ __forceinline__ void block_lookbacks(unsigned long long (&v)[K], uint32_t tile,
                                                       unsigned long long* const (&tiles)[K],
                                                       DeviceStatus* st) {
    static_assert(K <= kLookThreads / 32, "a warp for each value");
    __shared__ unsigned long long s_sum[K][kLookThreads / 32];
    __shared__ unsigned long long s_before[K];
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned long long incl[K];
#pragma unroll
    for (int i = 0; i < K; i++) {
        incl[i] = v[i];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned long long t = __shfl_up_sync(0xffffffffu, incl[i], d);
            if (lane >= (uint32_t)d) incl[i] += t;
        }
        if (lane == 31) s_sum[i][wid] = incl[i];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < K; i++) {
        if (wid != (uint32_t)i) continue;
        unsigned long long all = 0;
#pragma unroll
        for (int w = 0; w < kLookThreads / 32; w++) all += s_sum[i][w];
        const unsigned long long before = warp_lookback(all, tile, tiles[i], st);
        if (lane == 0) s_before[i] = before;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < K; i++) {
        v[i] = s_before[i] + incl[i] - v[i];
        for (uint32_t w = 0; w < wid; w++) v[i] += s_sum[i][w];
    }
}

// The same for one value.
static __device__ __forceinline__ unsigned long long block_lookback(unsigned long long v,
                                                                    uint32_t tile, LookState ls,
                                                                    DeviceStatus* st) {
    unsigned long long k[1] = {v};
    unsigned long long* const t[1] = {ls.tiles};
    block_lookbacks<1>(k, tile, t, st);
    return k[0];
}

// The last mark before this tile, by the same scheme (warp 0 of the block; the
// result in every lane): mine = the tile's last mark, 0 if it has none.  A
// tile with a mark of its own answers for all before it; the first has one.
static __device__ __forceinline__ unsigned long long warp_last_mark(unsigned long long mine,
                                                                    uint32_t tile,
                                                                    unsigned long long* tiles,
                                                                    DeviceStatus* st) {
    const uint32_t lane = threadIdx.x & 31;
    if (lane == 0) look_store(&tiles[tile], (mine ? kLookPrefix : kLookSum) | mine);
    unsigned long long found = 0;
    for (int64_t b = (int64_t)tile - 1; b >= 0; b -= 32) {
        const int64_t i = b - (int64_t)lane;
        const unsigned long long s = i >= 0 ? look_wait(&tiles[i], st) : kLookSum;
        const uint32_t full = __ballot_sync(0xffffffffu, (s >> 62) == 2ull);
        if (full) {
            found = __shfl_sync(0xffffffffu, s & kLookMask, __ffs(full) - 1);
            break;
        }
    }
    if (lane == 0 && !mine) look_store(&tiles[tile], kLookPrefix | found);
    return found;
}

// The same for one counter per thread: states of tile t at p[t * stride].
constexpr int kDigitLooks = 8;
static __device__ __forceinline__ unsigned long long digit_lookback(uint32_t v, uint32_t tile,
                                                                    unsigned long long* p,
                                                                    uint32_t stride,
                                                                    DeviceStatus* st) {
    if (tile == 0) {
        look_store(p, kLookPrefix | v);
        return 0;
    }
    look_store(p + (size_t)tile * stride, kLookSum | v);
    unsigned long long before = 0;
    for (int64_t t = (int64_t)tile - 1; t >= 0;) {
        // many states at once: their loads overlap
        unsigned long long s[kDigitLooks];
#pragma unroll
        for (int j = 0; j < kDigitLooks; j++)
            s[j] = t - j >= 0 ? look_load(p + (size_t)(t - j) * stride) : kLookPrefix;
        bool done = false;
#pragma unroll
        for (int j = 0; j < kDigitLooks; j++) {
            if (done) continue;
            if ((s[j] >> 62) == 0ull) s[j] = look_wait(p + (size_t)(t - j) * stride, st);
            before += s[j] & kLookMask;
            done = (s[j] >> 62) == 2ull;
        }
        if (done) break;
        t -= kDigitLooks;
    }
    look_store(p + (size_t)tile * stride, kLookPrefix | (before + v));
    return before;
}

}  // namespace vdb
