// Bucket sort: the default path (min_k = 0) of device sorts whose keys spread
// evenly enough. A merge level moves every item once through HBM and doubles the
// runs, a radix pass from the lowest digit up settles eight bits of the key; from the
// top down the array is cut into buckets that fit shared memory after
// log2(n / bucket) bits, 16 for 2^28 keys, and one more pass sorts every bucket
// whole. So a sort is two partition passes and a bucket pass (one partition pass up
// to 256 buckets) whatever the width of the key.
//
//   bk_sample_kernel  samples the keys of a segment, chooses the range that is
//                     cut into 2^(b1+b2) equal slices, and sees whether a slice
//                     is far too full
//   bk_hist_all_kernel, bk_sum_kernel, bk_list_kernel
//                     one segment of two levels: counts both levels' slices with one
//                     read; bucket sizes against what the last kernel can take; slice
//                     starts and the second level's tiles
//   bk_hist_kernel    else: counts a level's slices, one read
//   bk_scan_kernel    the same as sum and list, for one level (the first level of one
//                     segment: by the last CTA of bk_hist_kernel)
//   bk_pass_kernel    one partition level for keys, one read and one write
//   radix_pass_kernel the same for pairs, whose order has to be kept
//   bk_sort_kernel    one bucket per CTA, sorted in shared memory (64-bit keys:
//                     sb_sort_kernel, seg_buckets.cuh)
//
// Measured (one GB300): 2^28 uint32 keys 7.38 ms by merges, 3.79 by eight-bit radix
// passes, 2.63 by buckets (counting 0.22, partition 2 x 0.60, buckets 1.20); 2^27 uint64
// keys 8.44 by merges and 2.02 (0.20, 2 x 0.47, 0.85); 2^27 pairs 14.0 and 3.88 (0.33,
// 2 x 1.07, 1.38). A plain copy takes 0.32, 0.32 and 0.64 ms.
//
// A slice is a monotone function of the key (keys outside the sampled range
// fall into the end slices), so any data is sorted correctly as long as every
// bucket fits. Where one does not (heavy duplicates, clustered keys), *route is
// set on the device, the remaining kernels return at once, and what follows in the
// stream sorts the array instead (radix_host.cuh, Behind): the levels of the segmented
// bucket sort for 64-bit keys (seg_buckets.cuh; from the slices of the first level, where
// they are there already), radix passes for 32-bit keys (radix.cuh), for chunks of them
// merges or levels.
//
// Equal keys of keys-only items are identical, so their order does not matter:
// bk_pass_kernel takes places with shared-memory atomics, one CTA per tile in
// any order, and claims each slice's output range with one global atomic. No
// kernel here waits for another CTA. Each kernel starts while the last CTAs of the one
// before it run (programmatic dependent launch; no kernel lets the next one in earlier,
// its waiting CTAs would cost more than the launch: 2^20 uint32 keys 44 us with, 38
// without), so no pointer here is __restrict__ (no loads through the read-only path)
// and everything shared is read after grid_dep_wait().
#pragma once
#include <cstdint>

#include "bulk.cuh"
#include "common.cuh"
#include "radix.cuh"
#include "warp_sort.cuh"

namespace origami {

// *route: 0 buckets; 1 it gave up, the items are where they were; 2 it gave up, the
// first partition pass has moved the items to the other buffer.
enum BucketRoute : int { ROUTE_BUCKETS = 0, ROUTE_RADIX = 1, ROUTE_RADIX_MOVED = 2 };

template <class T>
struct BucketCfg;
template <>
struct BucketCfg<uint32_t> {
    static constexpr int NT = 256, IPT = 32, MINB = 3;        // partition tile: 8192 keys
    static constexpr int S_NT = 256, S_IPT = 24, S_MINB = 4;  // bucket: up to 6144 keys
    static constexpr int BINS = 4096;                         // bins of the bucket sort
    static constexpr int LOG_TARGET = 12;                     // mean bucket of 2048 to 4096 keys
};
template <>
struct BucketCfg<uint64_t> {
    static constexpr int NT = 256, IPT = 16, MINB = 3;
    static constexpr int S_NT = 256, S_IPT = 16, S_MINB = 4;
    static constexpr int BINS = 2048;
    static constexpr int LOG_TARGET = 11;
};
template <>
struct BucketCfg<KV64> {
    static constexpr int NT = 256, IPT = 16, MINB = 2;  // (radix_pass_kernel's tile)
    static constexpr int S_NT = 512, S_IPT = 8, S_MINB = 2;
    static constexpr int BINS = 2048;
    static constexpr int LOG_TARGET = 11;
};
template <class T>
struct BucketShape {
    using C = BucketCfg<T>;
    static constexpr bool STABLE = Traits<T>::kStable;
    static constexpr int TILE = C::NT * C::IPT;
    static constexpr size_t PASS_SMEM = (size_t)TILE * sizeof(T);
    static constexpr int CAP = C::S_NT * C::S_IPT;  // largest bucket
    // largest bin that neighbours settle (32: 4000 Zipf uint32 keys 22 us, 16: 18; 2^27
    // Zipf uint64 keys 3.76 and 3.28 ms)
    static constexpr int CROWDED = 16;
    static constexpr int FEW = 256;  // buckets up to here: ranked by comparison with all instead
    static constexpr int SETTLED = 33;  // items of a bin that a warp settles whatever their keys
    static constexpr int SIDE = STABLE ? 0 : CROWDED;  // guard keys on either side of the bucket
    static constexpr size_t KEYS_BYTES = (size_t)(CAP + 2 * SIDE) * sizeof(T);
    static constexpr size_t BIN_BYTES = (size_t)C::BINS * 4 + (STABLE ? (size_t)CAP * 2 : 0);  // bins, places (pairs)
    // crowded bins, behind them: their list; for every warp 32 places of a bin, and
    // (pairs) a bitmap of original places with its running counts
    static constexpr int WARPS = C::S_NT / 32, MOST_CROWDED = CAP / (CROWDED + 1);
    static constexpr int MAP_WORDS = STABLE ? CAP / 32 + CAP / 64 : 0;
    static constexpr size_t CROWD_BYTES = (size_t)WARPS * MAP_WORDS * 4 + ((size_t)MOST_CROWDED + WARPS * 32) * 2;
    // or what bins by splitters need (BkSplit), or the words of byte passes. (For pairs two
    // CTAs of 96 KB and little more just fit a shared memory of 196 KB; 1.2 KB more, and an
    // L1 of 28 KB slowed the scattered stores: 2^27 pairs 1.55 ms, not 1.38.)
    static constexpr size_t BYTE_BYTES = (size_t)(C::S_NT / 16) * RADIX_BINS * 4;
    static constexpr int SPLITTERS = 256;
    static constexpr size_t SPLIT_BYTES = SPLITTERS * sizeof(typename Traits<T>::Key) + (2 * SPLITTERS + 32) * 4 +
                                          (size_t)CAP * (STABLE ? 4 : 2) + (STABLE ? CAP / 32 + CAP / 32 * 48 : 64);
    static constexpr size_t MORE_BYTES = BIN_BYTES + CROWD_BYTES > BYTE_BYTES ? BIN_BYTES + CROWD_BYTES : BYTE_BYTES;
    static constexpr size_t SORT_SMEM = KEYS_BYTES + (SPLIT_BYTES > MORE_BYTES ? SPLIT_BYTES : MORE_BYTES);
    static_assert(TILE == RadixShape<T>::TILE || !STABLE, "pairs partition by radix_pass_kernel");
};
// keys sampled per segment; fewer up to one partition level (2^28 uint32 keys in chunks of
// 2^19: samples 0.10 and 0.04 ms)
constexpr int BK_SAMPLES = 8192, BK_FEW = 2048;
constexpr uint64_t BK_FEW_UP_TO = 1 << 20;
constexpr int BK_MAX_BITS = 16;      // slices of both levels
constexpr uint64_t BK_SELF_CLEAR = 1 << 17;  // bytes

// How a segment's keys map to slices: x = the key's distance from lo, scaled so
// that hi's fills 32 bits; slice = x * mul >> 32. mul is a multiple of 2^b2, so
// the first level's digit is x * (mul >> b2) >> 32.
template <class K>
struct SliceMap {
    K lo, hi;
    uint32_t mul;
    int c;
    __device__ __forceinline__ uint32_t scaled(K k) const {
        k = k < lo ? lo : (k > hi ? hi : k);
        k -= lo;
        if constexpr (sizeof(K) == 8)
            return (uint32_t)((k << c) >> 32);
        else
            return k << c;
    }
    // 2^(b1 + b2) slices of [lo, hi]
    __device__ __forceinline__ void set(K lo_, K hi_, int b1, int b2) {
        lo = lo_;
        hi = hi_;
        const K r = hi - lo;
        uint32_t x;
        if constexpr (sizeof(K) == 8) {
            c = r ? __clzll((long long)r) : 0;
            x = (uint32_t)((r << c) >> 32);
        } else {
            c = r ? __clz((int)r) : 0;
            x = r << c;
        }
        // x >= 2^31 (r == 0: one slice)
        mul = r ? (uint32_t)(((1ull << 32) << b1) / ((uint64_t)x + 1)) << b2 : 0u;
    }
};

// Items to the keys' unsigned order (32-bit keys are unsigned already).
template <class T>
__device__ __forceinline__ T bk_flip(const T& v, uint64_t xmask) {
    if constexpr (sizeof(typename Traits<T>::Key) == 4)
        return v;
    else
        return Traits<T>::flip(v, xmask);
}

// Digit of a partition level: the first level's is the slice without its low b2
// bits, the second's is those bits.
template <class T>
struct SliceDigit {
    SliceMap<typename Traits<T>::Key> map;  // mul as the level wants it (level())
    uint64_t xmask;
    uint32_t mask;
    __device__ __forceinline__ void level(const SliceMap<typename Traits<T>::Key>& m, int shift) {
        map = m;
        map.mul >>= shift;
    }
    __device__ __forceinline__ unsigned operator()(const T& v) const {
        return __umulhi(map.scaled(Traits<T>::key(bk_flip(v, xmask))), map.mul) & mask;
    }
};
// The same for radix_pass_kernel, with the slice starts of the scan.
template <class T>
struct SliceDigitStable : SliceDigit<T> {
    static constexpr bool kHeavy = false;  // no digit of most of the items: the sample gives up on such slices
    const SliceMap<typename Traits<T>::Key>* maps;
    uint32_t map_shift;
    const uint32_t* start;
    int shift, bits;
    __device__ __forceinline__ void enter(uint32_t seg) { this->level(maps[seg >> map_shift], shift); }
    __device__ __forceinline__ uint32_t count(uint32_t seg, int bin) const {
        if (bin >= (1 << bits)) return 0;
        const uint32_t* s = start + ((size_t)seg << bits) + bin;
        return s[1] - s[0];
    }
    __device__ __forceinline__ uint32_t first(uint32_t seg, uint64_t sbase, uint32_t*) const {
        const int bin = threadIdx.x;
        return bin < (1 << bits) ? start[((size_t)seg << bits) + bin] - (uint32_t)sbase : 0u;
    }
};

// One tile of the second level (written by bk_scan_kernel).
struct __align__(16) BkTile {
    uint64_t base, sbase;           // first item; the first-level bucket's first item
    uint32_t slen, seg, ti, cnt;    // the bucket's length and number; tile inside it; items
};

// Where a level's tiles are: level 1 cuts segments of equal length, level 2 the
// tiles listed by the scan.
struct BkListed {
    using Tile = RadixUniform::Tile;
    const BkTile* rec;
    const uint32_t* count;
    __device__ __forceinline__ uint32_t total(uint32_t) const { return *count; }
    template <int TILE>
    __device__ __forceinline__ Tile tile(uint32_t t) const {
        const BkTile r = rec[t];
        Tile q;
        q.base = r.base;
        q.sbase = r.sbase;
        q.slen = r.slen;
        q.seg = r.seg;
        q.ti = r.ti;
        q.cnt = (int)r.cnt;
        return q;
    }
};

// ---------------------------------------------------------------- sample ---
// One CTA per segment of len items (the last may be shorter). The range is the
// samples', widened by 1/512 at each end: of n evenly spread keys about n/8192
// lie outside the samples at either end.
template <class T>
__global__ void __launch_bounds__(1024) bk_sample_kernel(const T* in, uint64_t n, uint64_t len, uint64_t xmask, int b1,
                                                         int b2, uint64_t cap, SliceMap<typename Traits<T>::Key>* maps,
                                                         int* route, uint4* zero, uint32_t nzero) {
    using K = typename Traits<T>::Key;
    constexpr int PER = BK_SAMPLES / 1024;
    extern __shared__ __align__(16) uint32_t half[];  // 2^(b1+b2) 16-bit counters
    __shared__ K smin[32], smax[32];
    __shared__ SliceMap<K> map;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, bits = b1 + b2;
    const uint64_t base = (uint64_t)blockIdx.x * len;
    const uint64_t m = n - base < len ? n - base : len;
    const int ns = m <= BK_FEW_UP_TO ? BK_FEW : BK_SAMPLES;
    for (uint32_t i = tid; i < nzero; i += 1024) zero[i] = make_uint4(0, 0, 0, 0);
    K v[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        if (i * 1024 >= ns) {
            v[i] = v[0];
            continue;
        }
        // evenly spaced, each moved inside its stretch by a hash
        const uint32_t j = (uint32_t)(i * 1024 + tid);
        const uint64_t a = (m * j) / (uint32_t)ns;
        const uint32_t gap = (uint32_t)((m * (j + 1)) / (uint32_t)ns - a);
        const uint64_t p = a + __umulhi(j * 2654435761u, gap);
        v[i] = Traits<T>::key(bk_flip(in[base + (p < m ? p : m - 1)], xmask));
    }
    for (int i = tid; i < (1 << bits) / 2 + 1; i += 1024) half[i] = 0;
    K lo = v[0], hi = v[0];
#pragma unroll
    for (int i = 1; i < PER; ++i) {
        lo = v[i] < lo ? v[i] : lo;
        hi = v[i] > hi ? v[i] : hi;
    }
    auto reduce = [&] {
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            const K a = __shfl_xor_sync(0xFFFFFFFFu, lo, o), b = __shfl_xor_sync(0xFFFFFFFFu, hi, o);
            lo = a < lo ? a : lo;
            hi = b > hi ? b : hi;
        }
    };
    reduce();
    if (lane == 0) {
        smin[warp] = lo;
        smax[warp] = hi;
    }
    __syncthreads();
    if (warp == 0) {
        lo = smin[lane];
        hi = smax[lane];
        reduce();
        if (lane == 0) {
            const K add = (K)((hi - lo) / 512 + 1), top = (K)~(K)0;
            lo = lo > add ? (K)(lo - add) : (K)0;
            hi = top - hi > add ? (K)(hi + add) : top;
            map.set(lo, hi, b1, b2);
            maps[blockIdx.x] = map;
        }
    }
    __syncthreads();
    bool full = false;
    const SliceMap<K> mp = map;
    // far too full: at least 16 samples, and twice the largest bucket by estimate
    const uint32_t most = max(15u, (uint32_t)min((unsigned long long)(2 * cap * (uint32_t)ns / m), 60000ull));
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        if (i * 1024 >= ns) break;
        const uint32_t s = __umulhi(mp.scaled(v[i]), mp.mul);
        const uint32_t h = (atomicAdd(&half[s >> 1], (s & 1) ? 0x10000u : 1u) >> ((s & 1) * 16) & 0xFFFFu) + 1;
        full |= h > most;
    }
    if (__syncthreads_or(full) && tid == 0) *route = ROUTE_RADIX;
}

// ------------------------------------------------------------------ scan ---
// A segment's counts (h: the count of slice tid) become slice starts in start[] and
// cursor[], and either the next level's tiles (tiles2 given) or the check that every
// bucket fits. Every thread of the CTA calls it.
struct BkScan {
    uint32_t *start, *cursor;
    BkTile* tiles2;
    uint32_t* count2;
    int* route;
    int full_route;
    uint64_t n;
    uint32_t last_seg;
};
template <class T>
__device__ __forceinline__ void bk_scan_segment(const BkScan& to, uint32_t seg, uint32_t base, int bits, uint32_t h) {
    constexpr uint32_t TILE = BucketShape<T>::TILE;
    __shared__ uint32_t ws[RADIX_BINS / 32], ws2[RADIX_BINS / 32], at2;
    const int tid = threadIdx.x, nb = 1 << bits;
    const size_t at = ((size_t)seg << bits) + tid;
    const uint32_t s = base + radix_bin_scan<uint32_t>(h, ws);
    if (tid < nb) {
        to.start[at] = s;
        if (to.cursor) to.cursor[at] = s;
        if (seg == to.last_seg && tid == nb - 1) to.start[at + 1] = (uint32_t)to.n;
    }
    if (to.tiles2) {
        // the segment's tiles stand together in the list, bucket by bucket
        const uint32_t nt = (h + TILE - 1) / TILE;
        uint32_t t0 = radix_bin_scan<uint32_t>(nt, ws2);
        if (tid == RADIX_BINS - 1) at2 = atomicAdd(to.count2, t0 + nt);
        __syncthreads();
        t0 += at2;
        for (uint32_t i = 0; i < nt; ++i) {
            BkTile r;
            r.sbase = s;
            r.base = (uint64_t)s + (uint64_t)i * TILE;
            r.slen = h;
            r.seg = (seg << bits) + (uint32_t)tid;
            r.ti = i;
            r.cnt = h - i * TILE < TILE ? h - i * TILE : TILE;
            to.tiles2[t0 + i] = r;
        }
    } else if (h > (uint32_t)BucketShape<T>::CAP) {
        *to.route = to.full_route;
    }
}
// One CTA per segment of the level (256 threads, one slice each).
template <class T>
__global__ void __launch_bounds__(RADIX_BINS)
    bk_scan_kernel(const uint32_t* hist, int bits, const uint32_t* seg_start, uint64_t len, BkScan to) {
    const uint32_t seg = blockIdx.x;
    grid_dep_wait();
    if (__syncthreads_or(route_load(to.route) != ROUTE_BUCKETS)) return;  // (a CTA of this kernel may set it)
    const uint32_t h = threadIdx.x < (1u << bits) ? hist[((size_t)seg << bits) + threadIdx.x] : 0;
    bk_scan_segment<T>(to, seg, seg_start ? seg_start[seg] : (uint32_t)(seg * len), bits, h);
}

// ------------------------------------------------------------------ hist ---
// Counts of a level's slices: hist[seg << log2(mask+1) | digit]. The lanes of a
// warp spread over COPIES copies of the counters.
template <class T, class G>
__global__ void __launch_bounds__(512) bk_hist_kernel(const T* in, G geo, uint32_t tiles,
                                                      const SliceMap<typename Traits<T>::Key>* maps,
                                                      uint32_t map_shift, uint64_t xmask, int shift, int bits,
                                                      uint32_t* hist, const int* route, BkScan to, uint32_t* done) {
    using Sh = BucketShape<T>;
    constexpr int COPIES = 16, TILE = Sh::TILE, V = Vec<T>::N, STEPS = TILE / V / 512;
    static_assert(STEPS * V * 512 == TILE, "whole vector steps");
    __shared__ uint32_t cnt[RADIX_BINS * COPIES];
    const int tid = threadIdx.x, col = tid & (COPIES - 1), nb = 1 << bits;
    grid_dep_wait();
    if (route_load(route) != ROUTE_BUCKETS) return;
    const uint32_t total = geo.total(tiles);
    const uint32_t t0 = (uint32_t)((uint64_t)total * blockIdx.x / gridDim.x);
    const uint32_t t1 = (uint32_t)((uint64_t)total * (blockIdx.x + 1) / gridDim.x);
    if (t0 >= t1) return;
    for (int i = tid; i < nb * COPIES; i += 512) cnt[i] = 0;
    __syncthreads();
    auto flush = [&](uint32_t seg) {
        __syncthreads();
        for (int i = tid; i < nb; i += 512) {
            uint32_t s = 0;
#pragma unroll
            for (int c = 0; c < COPIES; ++c) {
                s += cnt[i * COPIES + c];
                cnt[i * COPIES + c] = 0;
            }
            if (s) atomicAdd(hist + ((size_t)seg << bits) + i, s);
        }
        __syncthreads();
    };
    uint32_t seg = 0xFFFFFFFFu;
    SliceDigit<T> dig;
    dig.xmask = xmask;
    dig.mask = (uint32_t)nb - 1;
    for (uint32_t t = t0; t < t1; ++t) {
        const auto q = geo.template tile<TILE>(t);
        if (q.seg != seg) {
            if (seg != 0xFFFFFFFFu) flush(seg);
            seg = q.seg;
            dig.level(maps[seg >> map_shift], shift);
        }
        const T* p = in + q.base;
        // (second-level buckets start anywhere: items, not vectors)
        if (((uintptr_t)p & 15) == 0 && q.cnt == TILE) {
            uint4 x[STEPS];
#pragma unroll
            for (int j = 0; j < STEPS; ++j) x[j] = reinterpret_cast<const uint4*>(p)[j * 512 + tid];
#pragma unroll
            for (int j = 0; j < STEPS; ++j) {
                const T* e = reinterpret_cast<const T*>(&x[j]);
#pragma unroll
                for (int k = 0; k < V; ++k) atomicAdd(&cnt[dig(e[k]) * COPIES + col], 1u);
            }
        } else {
#pragma unroll 8
            for (int i = tid; i < q.cnt; i += 512) atomicAdd(&cnt[dig(p[i]) * COPIES + col], 1u);
        }
    }
    if (seg != 0xFFFFFFFFu) flush(seg);
    if (!done) return;
    // one segment: the CTA that adds its counts last turns them into starts
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (tid == 0) last = atomicAdd(done, t1 - t0) + (t1 - t0) == total;
    __syncthreads();
    if (last) {
        __threadfence();
        bk_scan_segment<T>(to, 0, 0, bits, tid < nb ? look_load(hist + tid) : 0u);
    }
}

// ------------------------------------------------- both levels of a segment ---
// Counts the slices of both levels with one read: up to 65536 counters of 16 bits in
// shared memory, one CTA per SM, its counts to a row of its own. A counter that passes
// CAP makes the sort give up, and so none can run over in a sort that goes on. Where the
// 32 keys of a step share a slice (sorted input) one lane counts for all. 2^28 uint32
// keys: two reads 0.43 ms, this one 0.22 (atomics; the read alone 0.16), 2^27 uint64
// 0.44 and 0.20, 2^27 pairs 0.73 and 0.33.
template <class T>
__global__ void __launch_bounds__(1024)
    bk_hist_all_kernel(const T* in, uint64_t n, const SliceMap<typename Traits<T>::Key>* maps, uint64_t xmask, int bits,
                       uint32_t* rows, int* route) {
    constexpr int NT = 1024, V = Vec<T>::N, TILE = BucketShape<T>::TILE, STEPS = TILE / V / NT;
    constexpr uint32_t CAP = BucketShape<T>::CAP;
    static_assert(STEPS * V * NT == TILE, "whole vector steps");
    extern __shared__ __align__(16) uint32_t half[];
    const int tid = threadIdx.x, lane = tid & 31;
    const uint32_t words = 1u << (bits - 1);
    for (uint32_t i = tid; i < words; i += NT) half[i] = 0;
    grid_dep_wait();
    if (__syncthreads_or(route_load(route) != ROUTE_BUCKETS)) return;  // (a CTA of this kernel may set it)
    const SliceMap<typename Traits<T>::Key> map = maps[0];
    __syncthreads();
    bool over = false;
    auto slice = [&](const T& v) -> uint32_t { return __umulhi(map.scaled(Traits<T>::key(bk_flip(v, xmask))), map.mul); };
    auto add_to = [&](uint32_t s, uint32_t add) {
        const uint32_t sh = (s & 1u) * 16u;
        over |= ((atomicAdd(&half[s >> 1], add << sh) >> sh) & 0xFFFFu) >= CAP;
    };
    auto count = [&](const T& v, bool in) {
        const uint32_t s = slice(v);
        const uint32_t s0 = __shfl_sync(0xFFFFFFFFu, s, 0);
        uint32_t add = in ? 1u : 0u;
        if (__all_sync(0xFFFFFFFFu, in && s == s0)) add = lane == 0 ? 32u : 0u;
        if (add) add_to(s, add);
    };
    const uint64_t tiles = (n + TILE - 1) / TILE;
    const uint64_t t0 = tiles * blockIdx.x / gridDim.x, t1 = tiles * (blockIdx.x + 1) / gridDim.x;
    uint4 x[STEPS];
    auto fetch = [&](uint64_t t) {
        if ((t + 1) * TILE <= n) {
#pragma unroll
            for (int j = 0; j < STEPS; ++j) x[j] = reinterpret_cast<const uint4*>(in + t * TILE)[j * NT + tid];
        }
    };
    fetch(t0);
    for (uint64_t t = t0; t < t1; ++t) {
        if ((t + 1) * TILE <= n) {
            uint4 y[STEPS];
#pragma unroll
            for (int j = 0; j < STEPS; ++j) y[j] = x[j];
            if (t + 1 < t1) fetch(t + 1);
            // (a warp whose first keys share a slice looks for such steps)
            const uint32_t s = slice(*reinterpret_cast<const T*>(&y[0]));
            const bool plain = !__all_sync(0xFFFFFFFFu, s == __shfl_sync(0xFFFFFFFFu, s, 0));
#pragma unroll
            for (int j = 0; j < STEPS; ++j) {
                const T* e = reinterpret_cast<const T*>(&y[j]);
                if (plain) {
#pragma unroll
                    for (int q = 0; q < V; ++q) add_to(slice(e[q]), 1u);
                } else {
#pragma unroll
                    for (int q = 0; q < V; ++q) count(e[q], true);
                }
            }
        } else {
            for (uint64_t i = t * TILE; i < n; i += NT) count(in[i + tid < n ? i + tid : n - 1], i + tid < n);
        }
    }
    if (__syncthreads_or(over) && tid == 0) *route = ROUTE_RADIX;
    for (uint32_t i = tid; i < words; i += NT) rows[(size_t)blockIdx.x * words + i] = half[i];
}

// Sums the rows: one CTA per first-level slice (256 threads, up to 128 words). hist2: the
// second level's counts; hist1: the first level's.
template <class T>
__global__ void __launch_bounds__(256)
    bk_sum_kernel(const uint32_t* rows, uint32_t nrows, int b1, int b2, uint32_t* hist1, uint32_t* hist2, int* route) {
    __shared__ uint32_t lo2[128], hi2[128], total;
    const int tid = threadIdx.x, w = tid & 127, part = tid >> 7, nw = 1 << (b2 - 1);
    if (tid == 0) total = 0;
    grid_dep_wait();
    if (__syncthreads_or(route_load(route) != ROUTE_BUCKETS)) return;  // (a CTA of this kernel may set it)
    const size_t words = (size_t)1 << (b1 + b2 - 1);
    const uint32_t* p = rows + ((size_t)blockIdx.x << (b2 - 1)) + w;
    uint32_t lo = 0, hi = 0;
    if (w < nw) {
#pragma unroll 8
        for (uint32_t r = part; r < nrows; r += 2) {
            const uint32_t x = p[r * words];
            lo += x & 0xFFFFu;
            hi += x >> 16;
        }
    }
    if (part) {
        lo2[w] = lo;
        hi2[w] = hi;
    }
    __syncthreads();
    uint32_t sum = 0;
    bool over = false;
    if (!part && w < nw) {
        lo += lo2[w];
        hi += hi2[w];
        sum = lo + hi;
        over = lo > (uint32_t)BucketShape<T>::CAP || hi > (uint32_t)BucketShape<T>::CAP;
        reinterpret_cast<uint2*>(hist2 + ((size_t)blockIdx.x << b2))[w] = make_uint2(lo, hi);
    }
    sum = __reduce_add_sync(0xFFFFFFFFu, sum);
    if ((tid & 31) == 0 && sum) atomicAdd(&total, sum);
    if (__syncthreads_or(over) && tid == 0) *route = ROUTE_RADIX;
    if (tid == 0) hist1[blockIdx.x] = total;
}

// Starts, cursors and the second level's tiles: one CTA per first-level slice.
template <class T>
__global__ void __launch_bounds__(256)
    bk_list_kernel(uint64_t n, int b1, int b2, const uint32_t* hist1, const uint32_t* hist2, uint32_t* start1,
                   uint32_t* cursor1, uint32_t* start2, uint32_t* cursor2, BkTile* tiles2, uint32_t* count2,
                   const int* route) {
    constexpr uint32_t TILE = BucketShape<T>::TILE;
    __shared__ uint32_t ws[RADIX_BINS / 32], ws2[RADIX_BINS / 32], ws3[RADIX_BINS / 32], mine[3];
    const int tid = threadIdx.x, n1 = 1 << b1, n2 = 1 << b2;
    const uint32_t seg = blockIdx.x;
    grid_dep_wait();
    if (route_load(route) != ROUTE_BUCKETS) return;
    const uint32_t h1 = tid < n1 ? hist1[tid] : 0, nt = (h1 + TILE - 1) / TILE;
    const uint32_t s1 = radix_bin_scan<uint32_t>(h1, ws), t1 = radix_bin_scan<uint32_t>(nt, ws2);
    if (tid == (int)seg) {
        mine[0] = s1;
        mine[1] = h1;
        mine[2] = t1;
    }
    if (seg == 0 && tid < n1) {
        start1[tid] = s1;
        if (cursor1) cursor1[tid] = s1;
        if (tid == n1 - 1) {
            start1[n1] = (uint32_t)n;
            *count2 = t1 + nt;
        }
    }
    const uint32_t h2 = tid < n2 ? hist2[((size_t)seg << b2) + tid] : 0;
    const uint32_t r2 = radix_bin_scan<uint32_t>(h2, ws3);
    __syncthreads();
    const uint32_t base = mine[0], len = mine[1], at = mine[2];
    if (tid < n2) {
        start2[((size_t)seg << b2) + tid] = base + r2;
        if (cursor2) cursor2[((size_t)seg << b2) + tid] = base + r2;
        if (seg == (uint32_t)n1 - 1 && tid == n2 - 1) start2[(size_t)n1 << b2] = (uint32_t)n;
    }
    for (uint32_t i = tid; i * TILE < len; i += 256) {
        BkTile r;
        r.sbase = base;
        r.base = (uint64_t)base + (uint64_t)i * TILE;
        r.slen = len;
        r.seg = seg;
        r.ti = i;
        r.cnt = len - i * TILE < TILE ? len - i * TILE : TILE;
        tiles2[at + i] = r;
    }
}

// ------------------------------------------------------------------ pass ---
// One partition level of keys-only items: count the tile's digits, claim each
// digit's output range, place the items in digit order in shared memory, write
// them out run by run. Per 32 keys the shared-memory pipe takes three random
// accesses of 3.5 bank conflicts (count, place, store). Atomics of lanes with
// one digit would be serialised (31 cycles), so in a tile whose neighbours
// share digits (sorted or nearly sorted input: a warp's first step is uniform)
// one lane counts and places for all where a step is uniform.
template <class T, class G>
__global__ void __launch_bounds__(BucketCfg<T>::NT, BucketCfg<T>::MINB)
    bk_pass_kernel(const T* src, T* dst, G geo, uint32_t tiles, const SliceMap<typename Traits<T>::Key>* maps,
                   uint32_t map_shift, uint64_t xmask, int shift, int bits, uint32_t* cursor, uint32_t n,
                   const int* route) {
    using Sh = BucketShape<T>;
    constexpr int NT = Sh::C::NT, IPT = Sh::C::IPT, TILE = Sh::TILE;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* skeys = reinterpret_cast<T*>(smem_raw);
    __shared__ uint32_t tab[RADIX_BINS], goff[RADIX_BINS], ws[RADIX_BINS / 32];
    static_assert(NT == RADIX_BINS && IPT % 4 == 0, "one thread per slice; four digits to a register");
    const int tid = threadIdx.x, lane = tid & 31, nb = 1 << bits;
    tab[tid] = 0;
    grid_dep_wait();
    if (route_load(route) != ROUTE_BUCKETS) return;
    const uint32_t t = blockIdx.x;
    if (t >= geo.total(tiles)) return;
    const auto q = geo.template tile<TILE>(t);
    SliceDigit<T> dig;
    dig.level(maps[q.seg >> map_shift], shift);
    dig.xmask = xmask;
    dig.mask = (uint32_t)nb - 1;
    T v[IPT];
    uint32_t dp[IPT / 4];  // the items' digits
    const bool whole = q.cnt == TILE;
    const T* p = src + q.base + tid;
    if (whole) {
#pragma unroll
        for (int i = 0; i < IPT; ++i) v[i] = p[i * NT];
    } else {
#pragma unroll
        for (int i = 0; i < IPT; ++i) v[i] = src[q.base + min(i * NT + tid, q.cnt - 1)];
    }
#pragma unroll
    for (int i = 0; i < IPT; i += 4)
        dp[i / 4] = dig(v[i]) | dig(v[i + 1]) << 8 | dig(v[i + 2]) << 16 | dig(v[i + 3]) << 24;
    auto digit = [&](int i) -> uint32_t { return __byte_perm(dp[i / 4], 0, 0x4440 | (i & 3)); };
    const bool plain = whole && !__all_sync(0xFFFFFFFFu, digit(0) == __shfl_sync(0xFFFFFFFFu, digit(0), 0));
    const int mine = q.cnt - tid;
    __syncthreads();
    if (plain) {
#pragma unroll
        for (int i = 0; i < IPT; ++i) atomicAdd(&tab[digit(i)], 1u);
    } else {
#pragma unroll
        for (int i = 0; i < IPT; ++i) {
            const uint32_t d = digit(i), d0 = __shfl_sync(0xFFFFFFFFu, d, 0);
            const bool in = i * NT < mine;
            if (__all_sync(0xFFFFFFFFu, in && d == d0)) {
                if (lane == 0) atomicAdd(&tab[d], 32u);
            } else if (in) {
                atomicAdd(&tab[d], 1u);
            }
        }
    }
    __syncthreads();
    const uint32_t c = tab[tid];
    uint32_t g = 0;
    if (c) g = atomicAdd(cursor + ((size_t)q.seg << bits) + tid, c);
    const uint32_t start = radix_bin_scan<uint32_t>(c, ws);
    tab[tid] = start;
    __syncthreads();
    if (plain) {
#pragma unroll
        for (int i = 0; i < IPT; ++i) skeys[atomicAdd(&tab[digit(i)], 1u)] = v[i];
    } else {
#pragma unroll
        for (int i = 0; i < IPT; ++i) {
            const uint32_t d = digit(i), d0 = __shfl_sync(0xFFFFFFFFu, d, 0);
            const bool in = i * NT < mine;
            uint32_t r = 0;
            if (__all_sync(0xFFFFFFFFu, in && d == d0)) {
                if (lane == 0) r = atomicAdd(&tab[d], 32u);
                r = __shfl_sync(0xFFFFFFFFu, r, 0) + lane;
            } else if (in) {
                r = atomicAdd(&tab[d], 1u);
            }
            if (in) skeys[r] = v[i];
        }
    }
    goff[tid] = g - start;
    __syncthreads();
    // (o < n always holds while the input does not change under the sort)
    if (whole) {
#pragma unroll 8
        for (int i = 0; i < IPT; ++i) {
            const T x = skeys[i * NT + tid];
            const uint32_t o = goff[dig(x)] + (uint32_t)(i * NT + tid);
            if (o < n) dst[o] = x;
        }
    } else {
        for (int j = tid; j < q.cnt; j += NT) {
            const T x = skeys[j];
            const uint32_t o = goff[dig(x)] + (uint32_t)j;
            if (o < n) dst[o] = x;
        }
    }
}

// ------------------------------------------------------------ bucket sort ---
// Sorts one bucket per CTA in shared memory: the keys' range in the bucket is
// cut into BINS bins of equal width, about as many as there are items, and the
// items are placed bin by bin. A place then differs from the item's rank by the
// items of its own bin that stand on the wrong side of it, and bins are ordered,
// so an item is compared with its W neighbours on either side, W + 1 the largest
// bin of the bucket: conflict-free loads, no bin bounds, one trip count for the
// CTA. (Pairs compare original positions on equal keys and so are stable.)
// Crowded bins (heavy keys, a few distinct keys, or clustered ones): where every
// crowded bin holds one key only, keys are in order as placed. Other buckets take bins by
// splitters (bk_sort_crowded; uint32 keys of plain sorts byte passes over the keys'
// distance from the smallest).
template <class T>
__device__ __forceinline__ bool bk_before(const T& a, int ia, const T& b, int ib) {
    return less(a, b) || (!less(b, a) && ia < ib);
}

// Byte passes over the bucket in sk[0, cnt), as radix_pass_kernel ranks: every
// 16 lanes own a stretch of items and 256 words of `table`.
template <class T, int NT, int IPT>
__device__ __forceinline__ void bk_byte_passes(T* sk, uint32_t* table, uint32_t* ws, int cnt,
                                               typename Traits<T>::Key klo, int bytes) {
    constexpr int NG = NT / 16;
    const int tid = threadIdx.x, hl = tid & 15, grp = tid >> 4;
    const unsigned one = 1u << hl, lt = one - 1u;
    uint32_t* gt = table + grp * RADIX_BINS;
    const int i0 = grp * (16 * IPT) + hl;
    T w[IPT];
#pragma unroll 1
    for (int b = 0; b < bytes; ++b) {
#pragma unroll
        for (int i = 0; i < IPT; ++i)
            if (i0 + i * 16 < cnt) w[i] = sk[i0 + i * 16];
        uint4* z = reinterpret_cast<uint4*>(gt);
#pragma unroll
        for (int i = 0; i < RADIX_BINS / 64; ++i) z[i * 16 + hl] = make_uint4(0, 0, 0, 0);
        __syncwarp();
        auto digit = [&](int i) -> unsigned { return (unsigned)((Traits<T>::key(w[i]) - klo) >> (8 * b)) & 255u; };
#pragma unroll
        for (int i = 0; i < IPT; ++i)
            if (i0 + i * 16 < cnt) atomicAdd(&gt[digit(i)], 1u << 16);
        __syncthreads();
        uint32_t total = 0;
        if (tid < RADIX_BINS)
            for (int g = 0; g < NG; ++g) total += table[g * RADIX_BINS + tid] >> 16;
        uint32_t run = radix_bin_scan<uint32_t>(total, ws);
        if (tid < RADIX_BINS)
            for (int g = 0; g < NG; ++g) {
                const uint32_t c = table[g * RADIX_BINS + tid] >> 16;
                table[g * RADIX_BINS + tid] = run << 16;
                run += c;
            }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < IPT; ++i) {
            const bool in = i0 + i * 16 < cnt;
            const unsigned d = in ? digit(i) : 0;
            if (in) atomicOr(&gt[d], one);
            __syncwarp();
            const uint32_t x = gt[d], m = x & 0xFFFFu;
            const uint32_t r = (x >> 16) + __popc(m & lt);
            __syncwarp();
            if (in && (m >> hl) == 1u) gt[d] = (r + 1) << 16;
            __syncwarp();
            if (in) sk[r] = w[i];
        }
        __syncthreads();
    }
}

// The words a bucket sort shares beside its dynamic shared memory. (Both are found by
// name, also in functions that are not inlined: through pointer arguments the accesses
// could be generic ones.)
template <class T>
struct BucketSortShared {
    uint32_t ws[BucketCfg<T>::S_NT / 32];
    uint32_t rlo[2], rhi[2], widest, listed;
    int odd;  // pairs that leave: how many of BK_TRIED items share a deep bin with another key
};
template <class T>
__device__ __forceinline__ BucketSortShared<T>& bk_shared() {
    __shared__ BucketSortShared<T> s;
    return s;
}
__device__ __forceinline__ unsigned char* bk_smem() {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    return smem_raw;
}
// threadIdx.x; read anew for 64-bit keys, so that what is computed from it is not kept
// in registers over the sort (2^27 uint64 keys 0.85 ms instead of 1.00; 2^28 uint32
// keys 1.22 instead of 1.20).
template <class T>
__device__ __forceinline__ int bk_tid() {
    int t = threadIdx.x;
    if (sizeof(typename Traits<T>::Key) == 8) asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
    return t;
}
// One warp sorts a crowded bin, items [s, s + c) of the bucket, if at most 32 of
// them differ from the bin's commonest key (found in a sample of 32): the ranks of
// those by comparison with each other, the others in between. Keys are sorted in
// place. Pairs go to `out`, equal keys in the order of their original places: a
// bitmap of the places, one bit per item of the bucket, and its running counts.
template <class T>
__device__ __noinline__ bool bk_settle_bin(uint16_t* odd, T* sk, const uint16_t* si, uint32_t* map, int s, int c,
                                           T* out, uint64_t xout) {
    using K = typename Traits<T>::Key;
    constexpr bool ST = Traits<T>::kStable;
    constexpr int WORDS = BucketShape<T>::CAP / 32, PER = WORDS / 32;
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const K pick = Traits<T>::key(sk[s + c * lane / 32]);
    const unsigned same = __match_any_sync(0xFFFFFFFFu, pick);
    const unsigned best = __reduce_max_sync(0xFFFFFFFFu, (unsigned)__popc(same) << 5 | (unsigned)lane);
    const K h = __shfl_sync(0xFFFFFFFFu, pick, (int)(best & 31u));
    uint16_t* before = reinterpret_cast<uint16_t*>(map + WORDS);
    if constexpr (ST) {
#pragma unroll
        for (int i = 0; i < PER; ++i) map[lane * PER + i] = 0;
        __syncwarp();
    }
    int n = 0;  // items that differ
    for (int i0 = 0; i0 < c; i0 += 32) {
        const int i = i0 + lane;
        const bool in = i < c, is = in && Traits<T>::key(sk[s + i]) == h;
        const unsigned m = __ballot_sync(0xFFFFFFFFu, in && !is);
        if (n + __popc(m) > 32) return false;
        if (in && !is) odd[n + __popc(m & lt)] = (uint16_t)i;
        n += __popc(m);
        if constexpr (ST)
            if (is) atomicOr(&map[si[s + i] >> 5], 1u << (si[s + i] & 31));
    }
    __syncwarp();
    const bool mine = lane < n;
    T x = Traits<T>::max_item();
    int ix = lane;
    if (mine) {
        x = sk[s + odd[lane]];
        if constexpr (ST) ix = si[s + odd[lane]];
    }
    const K k = Traits<T>::key(x);
    int r = 0;
    for (int j = 0; j < n; ++j) {
        const K kj = __shfl_sync(0xFFFFFFFFu, k, j);
        const int ij = __shfl_sync(0xFFFFFFFFu, ix, j);
        r += kj < k || (kj == k && ij < ix) ? 1 : 0;
    }
    const int below = __popc(__ballot_sync(0xFFFFFFFFu, mine && k < h));
    const int at = s + (k < h ? r : c - n + r);
    if constexpr (ST) {
        int sum = 0;
#pragma unroll
        for (int i = 0; i < PER; ++i) sum += __popc(map[lane * PER + i]);
        int inc = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if (lane >= o) inc += u;
        }
        int run = inc - sum;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            before[lane * PER + i] = (uint16_t)run;
            run += __popc(map[lane * PER + i]);
        }
        __syncwarp();
        for (int i = lane; i < c; i += 32) {
            const T y = sk[s + i];
            const int iy = si[s + i];
            if (Traits<T>::key(y) == h)
                out[s + below + before[iy >> 5] + __popc(map[iy >> 5] & ((1u << (iy & 31)) - 1u))] = bk_flip(y, xout);
        }
        if (mine) out[at] = bk_flip(x, xout);
        __syncwarp();
    } else {
        for (int i = below + lane; i < below + c - n; i += 32) sk[s + i] = h;
        if (mine) sk[at] = x;
    }
    return true;
}
// Keys only: settles every crowded bin of the bucket that stands in its bins, and whether
// that could be done; by the whole CTA. (A call of its own, as bk_sort_crowded below. Zipf
// keys in groups of 5000, 2^25 in all: uint32 0.52 ms when such a bucket was loaded and put
// in its bins once more first, 0.38 now; uint64 1.22 and 0.95.)
template <class T>
__device__ __noinline__ bool bk_settle_keys() {
    using Sh = BucketShape<T>;
    constexpr int NT = Sh::C::S_NT, BINS = Sh::C::BINS;
    unsigned char* smem_raw = bk_smem();
    BucketSortShared<T>& sh = bk_shared<T>();
    T* sk = reinterpret_cast<T*>(smem_raw) + Sh::SIDE;
    const uint32_t* tab = reinterpret_cast<const uint32_t*>(smem_raw + Sh::KEYS_BYTES);
    uint16_t* odd = reinterpret_cast<uint16_t*>(smem_raw + Sh::KEYS_BYTES + Sh::BIN_BYTES);
    uint16_t* bins = odd + Sh::WARPS * 32;
    const int tid = threadIdx.x, warp = tid >> 5;
    if (tid == 0) sh.listed = 0;
    __syncthreads();
    for (int b = tid; b < BINS; b += NT)
        if (tab[b] - (b ? tab[b - 1] : 0u) > (uint32_t)Sh::CROWDED) bins[atomicAdd(&sh.listed, 1u)] = (uint16_t)b;
    __syncthreads();
    bool mixed = false;
    for (int k = warp; k < (int)sh.listed; k += Sh::WARPS) {
        const int b = bins[k], s = b ? (int)tab[b - 1] : 0;
        mixed |= !bk_settle_bin<T>(odd + warp * 32, sk, nullptr, nullptr, s, (int)tab[b] - s, nullptr, 0);
    }
    return !__syncthreads_or(mixed);
}
// Clears the bins; no barrier needed before bk_sort_bucket.
template <class T>
__device__ __forceinline__ void bk_sort_init() {
    BucketSortShared<T>& sh = bk_shared<T>();
    using C = BucketCfg<T>;
    uint32_t* tab = reinterpret_cast<uint32_t*>(bk_smem() + BucketShape<T>::KEYS_BYTES);
    const int tid = bk_tid<T>();
    if (tid < 2) {
        sh.rlo[tid] = 0xFFFFFFFFu;
        sh.rhi[tid] = 0;
        sh.widest = 1;
    }
#pragma unroll
    for (int i = 0; i < C::BINS / C::S_NT; ++i) tab[i * C::S_NT + tid] = 0;
}
constexpr int BK_TRIED = 64;  // items of a crowded bucket of pairs that are looked at
// What becomes of a bucket with crowded bins of several keys: byte passes; left as it is
// (false is returned; keys only: if a warp a bin can't settle them); pairs: settled by a
// warp each, and left if that fails.
enum BkCrowded { BK_BYTES, BK_LEAVE, BK_SETTLE };
// One bucket of cnt items (up to CAP), by the whole CTA. (src == out: in place.) xin
// and xout: the sign flips of keys read and written.
template <class T, BkCrowded CROWD>
__device__ __forceinline__ bool bk_sort_bucket(const T* src, T* out, int cnt, uint64_t xin, uint64_t xout) {
    unsigned char* smem_raw = bk_smem();
    BucketSortShared<T>& sh = bk_shared<T>();
    using Sh = BucketShape<T>;
    using K = typename Traits<T>::Key;
    constexpr int NT = Sh::C::S_NT, IPT = Sh::C::S_IPT, BINS = Sh::C::BINS;
    constexpr int CAP = Sh::CAP, BPT = BINS / NT;  // bins per thread of the scan
    constexpr uint32_t CROWDED = Sh::CROWDED;
    T* sk = reinterpret_cast<T*>(smem_raw) + Sh::SIDE;
    uint32_t* tab = reinterpret_cast<uint32_t*>(smem_raw + Sh::KEYS_BYTES);
    uint16_t* si = reinterpret_cast<uint16_t*>(tab + BINS);  // pairs: original places
    const int tid = bk_tid<T>(), lane = tid & 31, warp = tid >> 5;
    // crowded bins
    uint32_t* map = reinterpret_cast<uint32_t*>(smem_raw + Sh::KEYS_BYTES + Sh::BIN_BYTES) + warp * Sh::MAP_WORDS;
    uint16_t* odd = reinterpret_cast<uint16_t*>(smem_raw + Sh::KEYS_BYTES + Sh::BIN_BYTES + Sh::WARPS * Sh::MAP_WORDS * 4);
    uint16_t* bins = odd + Sh::WARPS * 32;
    if (CROWD == BK_SETTLE && tid == 0) sh.listed = 0;
    const int mine = cnt - tid;  // this thread's item i exists when i * NT < mine
    T v[IPT];
    const T* p = src + tid;
    // the range of the bucket's keys; 64-bit keys by their upper halves first
    auto hi32 = [](K k) -> uint32_t {
        if constexpr (sizeof(K) == 8) return (uint32_t)(k >> 32);
        return (uint32_t)k;
    };
#pragma unroll
    for (int i = 0; i < IPT; ++i)
        if (i * NT < mine) v[i] = bk_flip(p[i * NT], xin);
    uint32_t lo = 0xFFFFFFFFu, hi = 0;
#pragma unroll
    for (int i = 0; i < IPT; ++i)
        if (i * NT < mine) {
            const uint32_t x = hi32(Traits<T>::key(v[i]));
            lo = min(lo, x);
            hi = max(hi, x);
        }
    lo = __reduce_min_sync(0xFFFFFFFFu, lo);
    hi = __reduce_max_sync(0xFFFFFFFFu, hi);
    __syncthreads();
    if (lane == 0) {
        atomicMin(&sh.rlo[0], lo);
        atomicMax(&sh.rhi[0], hi);
    }
    __syncthreads();
    K klo, kr;
    lo = sh.rlo[0];
    hi = sh.rhi[0];
    if constexpr (sizeof(K) == 8) {
        if (lo == hi) {
            uint32_t a = 0xFFFFFFFFu, b = 0;
#pragma unroll
            for (int i = 0; i < IPT; ++i)
                if (i * NT < mine) {
                    const uint32_t x = (uint32_t)Traits<T>::key(v[i]);
                    a = min(a, x);
                    b = max(b, x);
                }
            a = __reduce_min_sync(0xFFFFFFFFu, a);
            b = __reduce_max_sync(0xFFFFFFFFu, b);
            if (lane == 0) {
                atomicMin(&sh.rlo[1], a);
                atomicMax(&sh.rhi[1], b);
            }
            __syncthreads();
            klo = ((K)lo << 32) | sh.rlo[1];
            kr = (K)(sh.rhi[1] - sh.rlo[1]);
        } else {
            klo = (K)lo << 32;
            kr = ((K)(hi - lo) << 32) | 0xFFFFFFFFu;
        }
    } else {
        klo = lo;
        kr = hi - lo;
    }
    if (kr == 0) {  // one key: the bucket is sorted
        if (src == out && xin == xout) return true;
#pragma unroll
        for (int i = 0; i < IPT; ++i)
            if (i * NT < mine) out[i * NT + tid] = bk_flip(v[i], xout);
        return true;
    }
    int c;
    uint32_t xr;
    if constexpr (sizeof(K) == 8) {
        c = __clzll((long long)kr);
        xr = (uint32_t)((kr << c) >> 32);
    } else {
        c = __clz((int)kr);
        xr = kr << c;
    }
    // bins of equal width; rounded down, and never past the last bin (xr >= 2^31)
    const uint32_t mul = (uint32_t)(((float)BINS * 4294967296.0f) / ((float)xr + 512.0f)) - 1u;
    auto bin = [&](K k) -> uint32_t {
        k -= klo;
        if constexpr (sizeof(K) == 8)
            return __umulhi((uint32_t)((k << c) >> 32), mul);
        else
            return __umulhi(k << c, mul);
    };
    uint32_t bp[(IPT + 1) / 2];  // the items' bins
#pragma unroll
    for (int i = 0; i < IPT; ++i)
        if (i * NT < mine) {
            const uint32_t b = bin(Traits<T>::key(v[i]));
            bp[i / 2] = (i & 1) ? __byte_perm(bp[i / 2], b, 0x5410) : b;
            atomicAdd(&tab[b], 1u);
        }
    __syncthreads();
    bool crowded = false;
    {
        uint32_t h[BPT], sum = 0, wide = 0;
        if constexpr (BPT % 4 == 0) {
#pragma unroll
            for (int i = 0; i < BPT; i += 4) {
                const uint4 x = reinterpret_cast<const uint4*>(tab)[(tid * BPT + i) / 4];
                h[i] = x.x;
                h[i + 1] = x.y;
                h[i + 2] = x.z;
                h[i + 3] = x.w;
            }
        } else {
#pragma unroll
            for (int i = 0; i < BPT; ++i) h[i] = tab[tid * BPT + i];
        }
#pragma unroll
        for (int i = 0; i < BPT; ++i) {
            const uint32_t x = h[i];
            crowded |= x > CROWDED;
            if (CROWD == BK_SETTLE && x > CROWDED) bins[atomicAdd(&sh.listed, 1u)] = (uint16_t)(tid * BPT + i);
            wide = max(wide, x > CROWDED ? 0u : x);
            h[i] = sum;
            sum += x;
        }
        wide = __reduce_max_sync(0xFFFFFFFFu, wide);
        if (lane == 0) atomicMax(&sh.widest, wide);
        uint32_t inc = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if (lane >= o) inc += u;
        }
        if (lane == 31) sh.ws[warp] = inc;
        crowded = __syncthreads_or(crowded);
        uint32_t first = inc - sum;
#pragma unroll
        for (int w = 0; w < NT / 32; ++w)
            if (w < warp) first += sh.ws[w];
        if constexpr (BPT % 4 == 0) {
#pragma unroll
            for (int i = 0; i < BPT; i += 4)
                reinterpret_cast<uint4*>(tab)[(tid * BPT + i) / 4] =
                    make_uint4(first + h[i], first + h[i + 1], first + h[i + 2], first + h[i + 3]);
        } else {
#pragma unroll
            for (int i = 0; i < BPT; ++i) tab[tid * BPT + i] = first + h[i];
        }
    }
    __syncthreads();
    if constexpr (CROWD == BK_LEAVE && Sh::STABLE)
        if (crowded) {
            bool other = false;
            if (tid < BK_TRIED) {  // (the first ones)
                const bool here = tid < cnt;
                const K k = here ? Traits<T>::key(v[0]) : 0;
                const uint32_t b = here ? bp[0] & 0xFFFFu : 0u;
                const int s = (int)tab[b], e = b + 1 < BINS ? (int)tab[b + 1] : cnt;
                const unsigned with = __match_any_sync(0xFFFFFFFFu, b) & ~__match_any_sync(0xFFFFFFFFu, k);
                other = here && with && e - s > Sh::SETTLED;
            }
            const int odd = __syncthreads_count(other);
            if (tid == 0) sh.odd = odd;
            return false;
        }
    static_assert(CROWD == BK_LEAVE || (CROWD == BK_SETTLE) == Sh::STABLE, "pairs are not in order as placed");
#pragma unroll
    for (int i = 0; i < IPT; ++i)
        if (i * NT < mine) {
            const uint32_t r = atomicAdd(&tab[__byte_perm(bp[i / 2], 0, (i & 1) ? 0x4432 : 0x4410)], 1u);
            sk[r] = v[i];
            if constexpr (Sh::STABLE) si[r] = (uint16_t)(i * NT + tid);
        }
    if constexpr (!Sh::STABLE) {
        if (tid < Sh::SIDE) {
            sk[-1 - tid] = 0;
            sk[cnt + tid] = Traits<T>::max_item();
        }
    }
    __syncthreads();
    // a bin's word is its end now, and so the start of the next
    if (crowded) {
        bool mixed = false;
        if constexpr (CROWD == BK_SETTLE) {
            for (int k = warp; k < (int)sh.listed; k += Sh::WARPS) {
                const int b = bins[k], s = b ? (int)tab[b - 1] : 0;
                mixed |= !bk_settle_bin<T>(odd + warp * 32, sk, si, map, s, (int)tab[b] - s, out, xout);
            }
        } else if constexpr (!Sh::STABLE) {
            // keys only: a crowded bin of equal keys is in order
            for (int j = tid; j < cnt; j += NT) {
                const uint32_t b = bin(Traits<T>::key(sk[j]));
                const uint32_t e = tab[b], s = b ? tab[b - 1] : 0;
                mixed |= e - s > CROWDED && sk[j] != sk[s];
            }
        }
        mixed = __syncthreads_or(mixed);
        if constexpr (CROWD == BK_LEAVE && !Sh::STABLE) mixed = mixed && (cnt <= Sh::FEW || !bk_settle_keys<T>());
        if (mixed) {
            if constexpr (CROWD != BK_BYTES) {
                if constexpr (CROWD == BK_SETTLE) {
                    // settled bins were written: in place, the items are put back
                    if (src == out) {
#pragma unroll
                        for (int i = 0; i < IPT; ++i)
                            if (i * NT < mine) out[i * NT + tid] = bk_flip(v[i], xin);
                    }
                    __syncthreads();
                }
                return false;
            } else {
#pragma unroll
                for (int i = 0; i < IPT; ++i)
                    if (i * NT < mine) sk[i * NT + tid] = v[i];
                __syncthreads();
                bk_byte_passes<T, NT, IPT>(sk, tab, sh.ws, cnt, klo, ((int)sizeof(K) * 8 - c + 7) / 8);
                for (int i = tid; i < cnt; i += NT) out[i] = bk_flip(sk[i], xout);
                return true;
            }
        }
    }
    if constexpr (Sh::STABLE) {
        for (int j = tid; j < cnt; j += NT) {
            const T x = sk[j];
            const uint32_t b = bin(Traits<T>::key(x));
            const int e = (int)tab[b], s = b ? (int)tab[b - 1] : 0;
            if (CROWD == BK_SETTLE && e - s > (int)CROWDED) continue;
            int r = s;
            if (e - s > 1) {
                const int ix = (int)si[j];
                for (int i = s; i < e; ++i) r += bk_before(sk[i], (int)si[i], x, ix) ? 1 : 0;
            }
            out[r] = bk_flip(x, xout);
        }
    } else {
        const int w = (int)sh.widest;
#pragma unroll 2
        for (int j = tid; j < cnt; j += NT) {
            const T x = sk[j];
            int r = j;
#pragma unroll 2
            for (int k = 1; k < w; ++k) {
                r += sk[j + k] < x ? 1 : 0;
                r -= sk[j - k] > x ? 1 : 0;
            }
            out[r] = bk_flip(x, xout);
        }
    }
    return true;
}

// Bins by splitters, for buckets whose crowded bins a warp each does not settle: 256 of the
// bucket's own keys are the splitters, and the keys equal to each have a bin of their own.
// Then the bins hold few items of different keys however the keys are spread, and each
// item's rank in its bin is counted; equal keys are in order as placed (pairs after their
// original places are ranked, many equal ones by a bitmap of the places, a warp a bin).
// Bounded by the search, eight steps of a random shared load a key, twice, and the ranks:
// 21 instructions an item in all, 55 % of issue slots. A bin that is wide all the same
// (samples that mislead) sends the bucket to byte passes.
// Those took every such bucket before, up to eight passes: groups of 200 log-uniform keys,
// 2^25 in all, uint32 11.9 ms and now 3.2, uint64 20.8 and 3.5, pairs 38.5 and 5.7; groups
// of 1000 3.0 / 1.2, 5.0 / 1.6, 9.1 / 1.9; 2^24 uint64 keys in clusters 1.78 and 0.88. (Tried:
// 512 splitters, groups of 200 twice as long, larger ones the same; merges through registers
// in shared memory, groups of 5000 3.0 ms instead of 2.5.)
template <class T>
struct BkSplit {
    using K = typename Traits<T>::Key;
    static constexpr int SPLITTERS = BucketShape<T>::SPLITTERS, BINS = 2 * SPLITTERS + 1;
    static constexpr int MANY = 64;  // equal pairs from here on: by bitmap
    static constexpr uint32_t WIDE = 256;
    static constexpr int CAP = BucketShape<T>::CAP, PLACES = BucketShape<T>::STABLE ? CAP : 1;
    static constexpr int MAPS = BucketShape<T>::STABLE ? 8 : 1, WORDS = BucketShape<T>::STABLE ? CAP / 32 : 1;
    K sp[SPLITTERS];
    uint32_t tab[BINS + 31];
    uint16_t bin[CAP];             // by original place
    uint16_t at[PLACES];           // pairs: original places
    uint16_t list[BucketShape<T>::STABLE ? CAP / MANY : 1];  // bins of many equal pairs
    uint32_t map[MAPS][WORDS];     // one bit per item of the bucket
    uint16_t before[MAPS][WORDS];  // its running counts
};
// (These are calls of their own, from the start: in line, or with the items
// kept in registers over them, they cost the other buckets registers, 2^27 pairs 1.4 and 1.8
// ms; which of them are calls was chosen by the registers that the others keep. 32-bit keys
// of plain sorts, whose byte passes are few, are better off with these in line: 2^28 keys
// 1.20 ms, with a call 1.38.)
template <class T>
__device__ __noinline__ void bk_sort_bytes(const T* src, T* out, int cnt, uint64_t xin, uint64_t xout) {
    using Sh = BucketShape<T>;
    __builtin_assume(__isGlobal(src));
    __builtin_assume(__isGlobal(out));
    T* sk = reinterpret_cast<T*>(bk_smem());
    uint32_t* table = reinterpret_cast<uint32_t*>(bk_smem() + Sh::KEYS_BYTES);
    constexpr int NT = Sh::C::S_NT;
    for (int i = threadIdx.x; i < cnt; i += NT) sk[i] = bk_flip(src[i], xin);
    __syncthreads();
    bk_byte_passes<T, NT, Sh::C::S_IPT>(sk, table, bk_shared<T>().ws, cnt, 0, (int)sizeof(typename Traits<T>::Key));
    for (int i = threadIdx.x; i < cnt; i += NT) out[i] = bk_flip(sk[i], xout);
}
template <class T>
__device__ __noinline__ void bk_sort_split(const T* src, T* out, int cnt, uint64_t xin, uint64_t xout) {
    using Sh = BucketShape<T>;
    using W = BkSplit<T>;
    using K = typename Traits<T>::Key;
    constexpr int NT = Sh::C::S_NT, NS = W::SPLITTERS;
    static_assert(Sh::KEYS_BYTES + sizeof(W) <= Sh::SORT_SMEM, "it fits");
    __builtin_assume(__isGlobal(src));
    __builtin_assume(__isGlobal(out));
    T* sk = reinterpret_cast<T*>(bk_smem());
    W& w = *reinterpret_cast<W*>(bk_smem() + Sh::KEYS_BYTES);
    BucketSortShared<T>& sh = bk_shared<T>();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    __syncthreads();
    if (cnt <= Sh::FEW) {
        // every item's rank by comparison with all
        T x;
        if (tid < cnt) sk[tid] = x = bk_flip(src[tid], xin);
        __syncthreads();
        if (tid < cnt) {
            int r = 0;
#pragma unroll 4
            for (int i = 0; i < tid; ++i) r += less(x, sk[i]) ? 0 : 1;
#pragma unroll 4
            for (int i = tid + 1; i < cnt; ++i) r += less(sk[i], x) ? 1 : 0;
            out[r] = bk_flip(x, xout);
        }
        return;
    }
    for (int i = tid; i < W::BINS; i += NT) w.tab[i] = 0;
    if (tid < NS) {
        // evenly spaced, each moved inside its stretch by a hash
        const int a = cnt * tid / NS, gap = cnt * (tid + 1) / NS - a;
        const int p = a + (int)__umulhi((uint32_t)tid * 2654435761u + 12345u, (uint32_t)gap);
        w.sp[tid] = Traits<T>::key(bk_flip(src[min(p, cnt - 1)], xin));
    }
    if (tid == 0) sh.widest = sh.listed = 0;
    __syncthreads();
    if (warp == 0) {
        K s[NS / 32];
#pragma unroll
        for (int k = 0; k < NS / 32; ++k) s[k] = w.sp[k * 32 + lane];
        warp_sort<K, NS / 32>(s, NS);
        __syncwarp();
#pragma unroll
        for (int k = 0; k < NS / 32; ++k) w.sp[lane * (NS / 32) + k] = s[k];
    }
    __syncthreads();
    // 2i: between splitters i-1 and i; 2i+1: equal to splitter i
    auto bin = [&](K k) -> uint32_t {
        uint32_t p = 0;
#pragma unroll
        for (int s = NS / 2; s; s >>= 1)
            if (w.sp[p + s - 1] < k) p += s;
        const K x = w.sp[p];
        return 2 * p + (x < k ? 2u : (x == k ? 1u : 0u));
    };
#pragma unroll 4
    for (int i = tid; i < cnt; i += NT) {
        const uint32_t b = bin(Traits<T>::key(bk_flip(src[i], xin)));
        w.bin[i] = (uint16_t)b;
        atomicAdd(&w.tab[b], 1u);
    }
    __syncthreads();
    // starts: thread t has the bins below and of splitter t, the last one also that above all
    static_assert(NS == RADIX_BINS, "one thread a splitter");
    uint32_t mixed = 0, pure = 0;
    if (tid < NS) {
        mixed = w.tab[2 * tid];
        pure = w.tab[2 * tid + 1];
    }
    const uint32_t first = radix_bin_scan<uint32_t>(mixed + pure, sh.ws);
    if (tid < NS) {
        w.tab[2 * tid] = first;
        w.tab[2 * tid + 1] = first + mixed;
        if (Sh::STABLE && pure > (uint32_t)W::MANY) w.list[atomicAdd(&sh.listed, 1u)] = (uint16_t)(2 * tid + 1);
        uint32_t wide = mixed;
        if (tid == NS - 1) {
            wide = max(wide, w.tab[2 * NS]);
            w.tab[2 * NS] = first + mixed + pure;
        }
        wide = __reduce_max_sync(0xFFFFFFFFu, wide);
        if (lane == 0) atomicMax(&sh.widest, wide);
    }
    __syncthreads();
    if (sh.widest > W::WIDE) {
        bk_sort_bytes<T>(src, out, cnt, xin, xout);
        return;
    }
#pragma unroll 4
    for (int i = tid; i < cnt; i += NT) {
        const uint32_t r = atomicAdd(&w.tab[w.bin[i]], 1u);
        sk[r] = bk_flip(src[i], xin);
        if constexpr (Sh::STABLE) w.at[r] = (uint16_t)i;
    }
    __syncthreads();
    // a bin's word is its end now, and so the start of the next
    if constexpr (Sh::STABLE) {
        constexpr int PER = W::WORDS / 32;
        if (warp < W::MAPS)
            for (int k = warp; k < (int)sh.listed; k += W::MAPS) {
                uint32_t* map = w.map[warp];
                const int b = w.list[k], s = (int)w.tab[b - 1], e = (int)w.tab[b];
#pragma unroll
                for (int i = 0; i < PER; ++i) map[lane * PER + i] = 0;
                __syncwarp();
                for (int i = s + lane; i < e; i += 32) atomicOr(&map[w.at[i] >> 5], 1u << (w.at[i] & 31));
                __syncwarp();
                int sum = 0;
#pragma unroll
                for (int i = 0; i < PER; ++i) sum += __popc(map[lane * PER + i]);
                int inc = sum;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int u = __shfl_up_sync(0xFFFFFFFFu, inc, o);
                    if (lane >= o) inc += u;
                }
                int run = inc - sum;
#pragma unroll
                for (int i = 0; i < PER; ++i) {
                    w.before[warp][lane * PER + i] = (uint16_t)run;
                    run += __popc(map[lane * PER + i]);
                }
                __syncwarp();
                for (int i = s + lane; i < e; i += 32) {
                    const int o = w.at[i];
                    out[s + w.before[warp][o >> 5] + __popc(map[o >> 5] & ((1u << (o & 31)) - 1u))] = bk_flip(sk[i], xout);
                }
                __syncwarp();
            }
    }
    for (int j = tid; j < cnt; j += NT) {
        const T x = sk[j];
        const uint32_t b = bin(Traits<T>::key(x));
        const int e = (int)w.tab[b], s = b ? (int)w.tab[b - 1] : 0;
        int r = s;
        if constexpr (Sh::STABLE) {
            if ((b & 1u) && e - s > W::MANY) continue;
            const int ix = (int)w.at[j];
            for (int i = s; i < e; ++i) r += bk_before(sk[i], (int)w.at[i], x, ix) ? 1 : 0;
        } else if (b & 1u) {
            r = j;
        } else {
            for (int i = s; i < j; ++i) r += sk[i] <= x ? 1 : 0;
            for (int i = j + 1; i < e; ++i) r += sk[i] < x ? 1 : 0;
        }
        out[r] = bk_flip(x, xout);
    }
}

// Crowded bins, each settled by a warp, and whether that was all.
template <class T>
__device__ __noinline__ bool bk_settle_bucket(const T* src, T* out, int cnt, uint64_t xin, uint64_t xout) {
    __builtin_assume(__isGlobal(src));
    __builtin_assume(__isGlobal(out));
    bk_sort_init<T>();
    const bool done = bk_sort_bucket<T, BucketShape<T>::STABLE ? BK_SETTLE : BK_LEAVE>(src, out, cnt, xin, xout);
    __syncthreads();
    return done;
}
// One bucket of a CTA that takes several.
template <class T>
__device__ __noinline__ void bk_sort_settled(const T* src, T* out, int cnt, uint64_t xin, uint64_t xout) {
    __syncthreads();
    if (!bk_settle_bucket<T>(src, out, cnt, xin, xout)) bk_sort_split<T>(src, out, cnt, xin, xout);
}
// A bucket that bk_sort_bucket<T, BK_LEAVE> left just now. Keys: by splitters. Pairs: where
// a quarter of 64 items share a bin of more items than a warp settles with one of 32 that
// has another key, those bins would not be settled. (2^25 pairs, groups of 200, keys spread
// over their logarithms: 5.7 ms, 8.3 if settling is tried first; Zipf keys in groups of 1000,
// which are settled, 1.31, by splitters 1.87. The test on items still in registers; read
// again for it here, Zipf groups took 1.47, chunks of 4096 0.086 instead of 0.078.)
template <class T>
__device__ __noinline__ void bk_sort_crowded(const T* src, T* out, int cnt, uint64_t xin, uint64_t xout) {
    __builtin_assume(__isGlobal(src));
    __builtin_assume(__isGlobal(out));
    static_assert(BucketShape<T>::STABLE, "pairs");
    __syncthreads();
    if (bk_shared<T>().odd >= BK_TRIED / 4 || !bk_settle_bucket<T>(src, out, cnt, xin, xout))
        bk_sort_split<T>(src, out, cnt, xin, xout);
}
template <class T>
__device__ __forceinline__ void bk_sort_left(const T* src, T* out, int cnt, uint64_t xin, uint64_t xout) {
    if constexpr (BucketShape<T>::STABLE)
        bk_sort_crowded<T>(src, out, cnt, xin, xout);
    else
        bk_sort_split<T>(src, out, cnt, xin, xout);
}

template <class T>
__global__ void __launch_bounds__(BucketCfg<T>::S_NT, BucketCfg<T>::S_MINB)
    bk_sort_kernel(const T* src, T* dst, const uint32_t* start, uint64_t xin, uint64_t xout, uint32_t n,
                   const int* route) {
    bk_sort_init<T>();
    grid_dep_wait();
    if (route_load(route) != ROUTE_BUCKETS) return;
    const uint32_t b0 = start[blockIdx.x], b1 = start[blockIdx.x + 1];
    if (b1 <= b0 || b1 > n || b1 - b0 > (uint32_t)BucketShape<T>::CAP) return;
    constexpr BkCrowded CROWD = sizeof(T) == 4 ? BK_BYTES : BK_LEAVE;
    if (!bk_sort_bucket<T, CROWD>(src + b0, dst + b0, (int)(b1 - b0), xin, xout))
        bk_sort_left<T>(src + b0, dst + b0, (int)(b1 - b0), xin, xout);
}

// A sort of one bucket: n items (up to CAP) by one CTA. (1000 uint32
// keys 20 us by the tile sort of the merges, 10 here; 4000 uint64 keys 24 and 12, pairs 29
// and 12.)
template <class T>
__global__ void __launch_bounds__(BucketCfg<T>::S_NT)
    bk_one_kernel(const T* src, T* dst, int n, uint64_t xin, uint64_t xout, int* err) {
    if (err && threadIdx.x == 0) *err = 0;
    bk_sort_init<T>();
    if (bk_sort_bucket<T, BucketShape<T>::STABLE ? BK_SETTLE : BK_LEAVE>(src, dst, n, xin, xout)) return;
    __syncthreads();
    if (sizeof(T) == 4)  // (four byte passes: one CTA is done in 28 us, by splitters in 46)
        bk_sort_bytes<T>(src, dst, n, xin, xout);
    else
        bk_sort_split<T>(src, dst, n, xin, xout);
}

// The first kernel of a merge sort: sorts every `tile` items (up to CAP). 2^24 uint64 keys in
// tiles of 4096: 0.32 ms by register and shared-memory merges (block_sort), 0.12 here; pairs
// 0.51 (tiles of 2048) and 0.17.
template <class T>
__global__ void __launch_bounds__(BucketCfg<T>::S_NT, BucketCfg<T>::S_MINB)
    bk_tile_kernel(const T* in, T* out, uint64_t n, uint32_t tile, uint64_t xin, uint64_t xout, int* err) {
    const uint64_t base = (uint64_t)blockIdx.x * tile;
    const int cnt = n - base < tile ? (int)(n - base) : (int)tile;
    if (blockIdx.x == 0 && threadIdx.x == 0) *err = 0;
    bk_sort_init<T>();
    if (!bk_sort_bucket<T, BK_LEAVE>(in + base, out + base, cnt, xin, xout))
        bk_sort_left<T>(in + base, out + base, cnt, xin, xout);
}

}  // namespace origami
