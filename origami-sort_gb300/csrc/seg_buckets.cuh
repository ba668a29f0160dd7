// Segmented sorts by buckets: the default path for segments given by a device
// array of offsets. A merge level moves every item once through HBM and doubles
// the runs; a partition level moves every item once and cuts every segment into
// up to 256 slices, so one level and a pass over buckets that fit shared memory
// sort segments of up to a million items, two segments of any size.
//
//   sb_plan_kernel    short segments become buckets, the others the first
//                     level's segments
//   per level, over all segments of the level together:
//   sb_sample_kernel  samples a segment's keys and decides how it is cut; lists
//                     the segment's tiles
//   sb_hist_kernel    counts every segment's slices, one read; the last CTA of a
//                     segment scans them and hands the slices on: groups that fit
//                     become buckets, larger slices segments of the next level
//   sb_pass_kernel    moves the items (keys), one read and one write;
//   sb_stable_pass_kernel  the same for pairs, whose order has to be kept
//   then
//   sb_sort_kernel    sorts every bucket in shared memory
//
// The same levels stand behind the plain bucket sort of 64-bit keys (buckets.cuh), for
// keys that it gives up on.
//
// How a segment is cut. Its keys' range, from the sample, in 256 slices of equal
// width: a subtraction and a multiplication per key. Where one slice would take
// too many of the samples because of one key, that key gets a slice of its
// own, which needs no sorting. Where slices are uneven beyond that (clusters,
// several heavy keys), 127 sampled keys are the splitters instead, each with a
// slice of its own for the keys equal to it: seven steps of search per key, but
// slices of bounded size for any keys. All three are monotone functions of the
// key, so the sample decides only how even the slices are, never the result.
// Too many: 1/8 of the samples, and what the levels that follow would not cut into
// buckets by splitters. (With 1/8 alone clusters in clusters of 11 % of the keys
// left slices longer than a bucket: 838,000 uint64 keys 1.08 ms instead of 0.13, 2^27
// 19.3 instead of 3.45, by merges 8.4.)
//
// Segment lengths are on the device, so every list is made there: the host
// launches a fixed sequence (as many levels as one segment of all items may
// need by splitters; a level without segments returns at once) and never waits.
// Slices of the last level that still do not fit, possible only when samples
// mislead, are sorted by one CTA each in global memory.
//
// Equal keys of keys-only items are identical, so their order does not matter:
// sb_pass_kernel takes places with shared-memory atomics, tiles in any order, and
// claims each slice's output range with one global atomic; nothing waits for
// another CTA. Pairs are placed stably with a look-back over the tiles before
// (sb_stable_pass_kernel). Every wait (look-back, bulk copies) is bounded.
//
// The kernels overlap as the plain bucket sort's do: no pointer here is __restrict__,
// and everything shared is read after grid_dep_wait().
#pragma once
#include <cstdint>
#include <type_traits>

#include "buckets.cuh"

namespace origami {

constexpr int SB_SPLITTERS = 127;  // two slices each, and one above them
constexpr int SB_SAMPLES = 2048;   // keys sampled per segment
constexpr int SB_MAX_LEVELS = 4;
// A level by splitters cuts any segment by this: a slice is 16 of the samples, 1/128 of the
// segment, give or take a quarter.
constexpr int SB_SURE_BITS = 6;

// The tiles of a level's segments: 6144 uint32 keys, 4096 uint64 keys or pairs.
// (uint32: 8192 keys at three CTAs per SM pass 2^28 in 0.66 ms, 6144 at four in
// 0.62; 4096 at five in 0.84.)
template <class T>
struct SegBucketCfg;
template <>
struct SegBucketCfg<uint32_t> {
    static constexpr int NT = 256, IPT = 24, MINB = 4;
};
template <>
struct SegBucketCfg<uint64_t> {
    static constexpr int NT = 256, IPT = 16, MINB = 3;
};
template <>
struct SegBucketCfg<KV64> {
    static constexpr int NT = 256, IPT = 16, MINB = 2;
};
template <class T>
struct SegBucketShape {
    using C = SegBucketCfg<T>;
    using Sort = BucketShape<T>;  // the buckets' shape
    static constexpr bool STABLE = Traits<T>::kStable;
    static constexpr int TILE = C::NT * C::IPT;
    static constexpr int CAP = Sort::CAP;
    // partition: the tile; pairs also 256 words for every 16 lanes
    static constexpr size_t TILE_BYTES = (size_t)TILE * sizeof(T);
    static constexpr int GROUPS = C::NT / 16;
    static constexpr size_t PASS_SMEM = TILE_BYTES + (STABLE ? (size_t)GROUPS * RADIX_BINS * 4 : 0);
    // counting: keys arrive in two stages (a tile and the 16-byte chunks that
    // enclose it), pairs are read directly
    static constexpr size_t STAGE_BYTES = (TILE_BYTES + 16 + 127) & ~(size_t)127;
    static constexpr size_t HIST_SMEM = STABLE ? 0 : 2 * STAGE_BYTES;
};

// The two buffers of a sort. Level l moves the items from d to tmp where l is even and
// back where it is odd; behind a bucket sort that gave up after its first partition the
// other way round. The result is wanted in d or tmp.
template <class T>
struct SbBuffers {
    T *d, *tmp;
    const int* route;  // or null
    bool want_tmp;
    __device__ __forceinline__ bool moved() const { return route && route_load(route) == ROUTE_RADIX_MOVED; }
    __device__ __forceinline__ bool from_tmp(int level) const { return ((level & 1) != 0) != moved(); }
    __device__ __forceinline__ T* want() const { return want_tmp ? tmp : d; }
};
// The first level's segments behind a plain bucket sort (buckets.cuh): none where it
// went on; else nseg segments of len of n items, or, after its first partition, the
// `slices` of that.
struct SbGiven {
    const int* route;  // null: it was left out
    const uint32_t* start1;
    uint64_t n, len;
    uint32_t nseg, slices;
};

// ------------------------------------------------------------------ lists ---
struct SbSeg {  // a segment of a level
    uint64_t base, len;
};
struct __align__(16) SbTile {  // one tile of a level
    uint64_t base, sbase, slen;  // first item; the segment's first item and length
    uint32_t seg, cnt;           // the segment's number in the level; items
};
struct __align__(16) SbRec {  // one bucket
    uint64_t base, what;      // first item; length and flags
    static constexpr uint64_t TMP = 1ull << 62;   // the items are in tmp (else in d)
    static constexpr uint64_t SLOW = 1ull << 60;  // does not fit: sorted in global memory
    static constexpr uint64_t LEN = (1ull << 60) - 1;
};
// Counters, 0 at launch: a part of the sort's 256-byte tail, whose first word is
// the error word.
struct SbCounts {
    int err;
    uint32_t pad[15];
    uint32_t recs, slow, segs[SB_MAX_LEVELS + 1], tiles[SB_MAX_LEVELS], claim[SB_MAX_LEVELS];
};
static_assert(sizeof(SbCounts) <= 256, "the tail");

// A counter from L2: kernels overlap, and an earlier one of them may write it.
__device__ __forceinline__ uint32_t count_load(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// How a segment's keys map to slices. Linear: x = the key's distance from lo,
// scaled so that hi's fills 32 bits; slice = x * mul >> 32. HEAVY: 254 linear
// slices and one for the keys equal to `heavy`, between those below and above it.
// SEARCH: by splitters.
enum SbMode : uint32_t { SB_LINEAR = 0, SB_HEAVY = 1, SB_SEARCH = 2 };
template <class K>
struct SbMap {
    K lo, hi, heavy;
    uint32_t mul;
    int c;
    uint32_t mode, heavy_slice;
    __device__ __forceinline__ uint32_t linear(K k) const {
        k = k < lo ? lo : (k > hi ? hi : k);
        k -= lo;
        uint32_t x;
        if constexpr (sizeof(K) == 8)
            x = (uint32_t)((k << c) >> 32);
        else
            x = k << c;
        return __umulhi(x, mul);
    }
    __device__ __forceinline__ uint32_t with_heavy(K k) const {
        return linear(k) + (k >= heavy ? 1u : 0u) + (k > heavy ? 1u : 0u);
    }
    __device__ __forceinline__ void set(K lo_, K hi_, uint32_t slices) {
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
        mul = r ? (uint32_t)(((1ull << 32) * slices) / ((uint64_t)x + 1)) : 0u;
    }
    // a slice of equal keys?
    __device__ __forceinline__ bool pure(uint32_t slice) const {
        return mode == SB_SEARCH ? (slice & 1u) != 0 : mode == SB_HEAVY && slice == heavy_slice;
    }
};
// Slice by splitters sp[0 .. 127] (ascending, the last one the largest key): 2i
// for keys between splitters i-1 and i, 2i+1 for keys equal to splitter i.
template <class K>
__device__ __forceinline__ uint32_t sb_search(K k, const K* sp) {
    uint32_t p = 0;
#pragma unroll
    for (int s = 64; s; s >>= 1)
        if (sp[p + s - 1] < k) p += s;
    return 2 * p + (sp[p] == k ? 1u : 0u);
}
template <class T>
struct SbDigit {
    using K = typename Traits<T>::Key;
    SbMap<K> map;
    uint64_t xmask;
    const K* sp;  // shared memory, 128 keys
    template <uint32_t MODE>
    __device__ __forceinline__ uint32_t by(const T& v) const {
        const K k = Traits<T>::key(bk_flip(v, xmask));
        if constexpr (MODE == SB_LINEAR)
            return map.linear(k);
        else if constexpr (MODE == SB_HEAVY)
            return map.with_heavy(k);
        else
            return sb_search<K>(k, sp);
    }
    // f(mode) with the segment's mode as a compile-time constant
    template <class F>
    __device__ __forceinline__ void with_mode(F&& f) const {
        if (map.mode == SB_LINEAR)
            f(std::integral_constant<uint32_t, SB_LINEAR>());
        else if (map.mode == SB_HEAVY)
            f(std::integral_constant<uint32_t, SB_HEAVY>());
        else
            f(std::integral_constant<uint32_t, SB_SEARCH>());
    }
};

// ------------------------------------------------------------------- plan ---
// Segmented sorts, one thread per segment: short segments are buckets as they
// are, the others segments of the first level. A bad segment (decreasing offsets
// or past the buffer) is reported and left out.
template <class T>
__global__ void sb_plan_kernel(const uint64_t* off, uint32_t nseg, uint64_t n, SbSeg* list, uint32_t most, SbRec* recs,
                               SbCounts* cn) {
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    uint64_t a = 0, len = 0;
    if (s < nseg) {
        a = off[s];
        const uint64_t b = off[s + 1];
        if (a <= b && b <= n)
            len = b - a;
        else
            atomicExch(&cn->err, ERR_BAD_OFFSETS);
    }
    const bool big = len > (uint64_t)SegBucketShape<T>::CAP, small = len > 1 && !big;
    const unsigned lane = threadIdx.x & 31, mb = __ballot_sync(0xFFFFFFFFu, big), ms = __ballot_sync(0xFFFFFFFFu, small);
    uint32_t ib = 0, is = 0;
    if (lane == 0) {
        if (mb) ib = atomicAdd(&cn->segs[0], (uint32_t)__popc(mb));
        if (ms) is = atomicAdd(&cn->recs, (uint32_t)__popc(ms));
    }
    ib = __shfl_sync(0xFFFFFFFFu, ib, 0) + __popc(mb & ((1u << lane) - 1u));
    is = __shfl_sync(0xFFFFFFFFu, is, 0) + __popc(ms & ((1u << lane) - 1u));
    if (big && ib < most) list[ib] = SbSeg{a, len};
    if (small) recs[is] = SbRec{a, len};
}

// ----------------------------------------------------------------- sample ---
// One CTA per segment of the level (given.nseg: the first one behind a bucket sort;
// segments that fit a bucket become one here). The linear range is the samples',
// widened by 1/512 at each end. more: the levels that follow this one.
template <class T, class S>
__global__ void __launch_bounds__(512)
    sb_sample_kernel(SbBuffers<T> buf, int level, int more, SbGiven given, const SbSeg* list, uint32_t* count, uint64_t xmask,
                     SbMap<typename Traits<T>::Key>* maps, typename Traits<T>::Key* splitters, S* hist, uint32_t* done,
                     SbTile* tiles, uint32_t* tile_count, SbRec* recs, uint32_t* rec_count, const int* err) {
    using K = typename Traits<T>::Key;
    constexpr int NT = 512, PER = SB_SAMPLES / NT;
    constexpr uint32_t TILE = SegBucketShape<T>::TILE;
    // longest slice, by the samples, that the levels that follow are sure to cut (half a
    // bucket where there are none: a share of 32 samples is one of 18 to 46)
    constexpr int CAP = SegBucketShape<T>::CAP;
    const uint64_t sure = more ? (uint64_t)(CAP * 3 / 4) << (SB_SURE_BITS * more) : (uint64_t)(CAP / 2);
    __shared__ K smp[SB_SAMPLES];
    __shared__ K smin[NT / 32], smax[NT / 32], scand;
    __shared__ uint32_t cnt[RADIX_BINS];
    __shared__ SbMap<K> smap;
    __shared__ uint32_t stile, sid;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    grid_dep_wait();
    // (segments that overlap would not fit the lists)
    uint32_t total;
    bool slices = false;
    if (given.nseg) {
        const int route = given.route ? route_load(given.route) : (int)ROUTE_RADIX;
        slices = route == ROUTE_RADIX_MOVED;
        total = route == ROUTE_BUCKETS ? 0u : (slices ? given.slices : given.nseg);
    } else {
        total = count_load((const uint32_t*)err) == ERR_BAD_OFFSETS ? 0u : count_load(count);
    }
    if (blockIdx.x >= total) return;
    const T* src = buf.from_tmp(level) ? buf.tmp : buf.d;
    for (uint32_t at = blockIdx.x; at < total; at += gridDim.x) {
        SbSeg q;
        uint32_t sg = at;
        if (given.nseg) {
            q.base = slices ? given.start1[at] : at * given.len;
            q.len = (slices ? given.start1[at + 1] : (given.n - q.base < given.len ? given.n : q.base + given.len)) - q.base;
            const bool fits = q.len <= (uint64_t)SegBucketShape<T>::CAP;
            if (tid == 0) {
                if (!fits)
                    sid = atomicAdd(count, 1u);
                else if (q.len)
                    recs[atomicAdd(rec_count, 1u)] = SbRec{q.base, q.len | (slices ? SbRec::TMP : 0)};
            }
            if (fits) continue;
            __syncthreads();
            sg = sid;
        } else {
            q = list[at];
        }
        K v[PER], lo, hi;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            // evenly spaced, each moved inside its stretch by a hash
            const uint32_t j = (uint32_t)(i * NT + tid);
            const uint64_t a = q.len * j / SB_SAMPLES;
            const uint32_t gap = (uint32_t)min(q.len * (j + 1) / SB_SAMPLES - a, (uint64_t)0xFFFFFFFFu);
            const uint64_t p = a + __umulhi(j * 2654435761u + 12345u, gap);
            v[i] = Traits<T>::key(bk_flip(src[q.base + (p < q.len ? p : q.len - 1)], xmask));
        }
        if (tid < RADIX_BINS) {
            cnt[tid] = 0;
            hist[(size_t)sg * RADIX_BINS + tid] = 0;
        }
        lo = hi = v[0];
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
        const uint32_t nt = (uint32_t)((q.len + TILE - 1) / TILE);
        if (tid == NT - 1) {
            stile = atomicAdd(tile_count, nt);
            done[sg] = 0;
        }
        __syncthreads();
        if (warp == 0) {
            lo = smin[lane & (NT / 32 - 1)];
            hi = smax[lane & (NT / 32 - 1)];
            reduce();
            if (lane == 0) {
                const K add = (K)((hi - lo) / 512 + 1), top = (K)~(K)0;
                lo = lo > add ? (K)(lo - add) : (K)0;
                hi = top - hi > add ? (K)(hi + add) : top;
                smap.set(lo, hi, RADIX_BINS);
            }
        }
        __syncthreads();
        SbMap<K> map = smap;
        map.mode = SB_LINEAR;
        map.heavy = 0;
        map.heavy_slice = 0;
        bool full = false;
        const uint32_t most = (uint32_t)min((uint64_t)(SB_SAMPLES / 8), SB_SAMPLES * sure / q.len);
#pragma unroll
        for (int i = 0; i < PER; ++i)
            if (atomicAdd(&cnt[map.linear(v[i])], 1u) >= most) {
                full = true;
                scand = v[i];  // a key of a crowded slice (any of them)
            }
        if (__syncthreads_or(full)) {
            // one heavy key, and even slices but for it?
            map.set(map.lo, map.hi, RADIX_BINS - 2);
            map.heavy = scand;
            if (tid < RADIX_BINS) cnt[tid] = 0;
            __syncthreads();
            full = false;
#pragma unroll
            for (int i = 0; i < PER; ++i)
                if (v[i] != map.heavy) full |= atomicAdd(&cnt[map.linear(v[i])], 1u) >= most;
            map.mode = __syncthreads_or(full) ? SB_SEARCH : SB_HEAVY;
            map.heavy_slice = map.linear(map.heavy) + 1;
        }
        if (tid == 0) maps[sg] = map;
        if (map.mode == SB_SEARCH) {
            // sort the samples (bitonic), 127 of them are the splitters
#pragma unroll
            for (int i = 0; i < PER; ++i) smp[i * NT + tid] = v[i];
            __syncthreads();
            for (int k = 2; k <= SB_SAMPLES; k <<= 1)
                for (int s = k >> 1; s; s >>= 1) {
                    for (int w = tid; w < SB_SAMPLES / 2; w += NT) {
                        const int a = (w / s) * 2 * s + (w & (s - 1));
                        const int b = s == k >> 1 ? a ^ (k - 1) : a + s;
                        const K x = smp[a], y = smp[b];
                        if (y < x) {
                            smp[a] = y;
                            smp[b] = x;
                        }
                    }
                    __syncthreads();
                }
            if (tid <= SB_SPLITTERS)
                splitters[(size_t)sg * (SB_SPLITTERS + 1) + tid] =
                    tid < SB_SPLITTERS ? smp[(tid + 1) * (SB_SAMPLES / (SB_SPLITTERS + 1)) - 1] : (K)~(K)0;
        }
        const uint32_t t0 = stile;
        for (uint32_t i = tid; i < nt; i += NT) {
            SbTile r;
            r.sbase = q.base;
            r.slen = q.len;
            r.base = q.base + (uint64_t)i * TILE;
            r.seg = sg;
            const uint64_t rest = q.len - (uint64_t)i * TILE;
            r.cnt = rest < TILE ? (uint32_t)rest : TILE;
            tiles[t0 + i] = r;
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------- hist ---
// Where the slices of a level go: the next level's list (none: the last level)
// and the buckets. Buckets lie in the level's output buffer, `flags` says which
// one that is; stay: it is also the buffer the result is wanted in.
struct SbHandOn {
    SbSeg* next;
    uint32_t* next_count;
    SbRec* recs;
    uint32_t *slow, *slow_count;
    uint32_t* rec_count;
    uint64_t flags;  // (set by the kernel)
    bool stay;       // equal keys need not be written again where they are wanted
};

// Turns a segment's counts (h: the count of slice tid, threads below 256) into
// slice starts, in place, and hands the slices on. Slices are grouped: neighbours
// of up to CAP/2 items, m the longest, form a bucket where they start in the same
// stretch of the segment; stretches are equal and at most CAP - m items long. Longer
// slices stand alone. Every thread
// of the CTA calls it.
template <class T, class S, int NT, class Map>
__device__ __forceinline__ void sb_hand_on(const SbTile& q, S h, const Map& map, S* row, const SbHandOn& to) {
    constexpr int CAP = SegBucketShape<T>::CAP, W = CAP / 2;
    __shared__ S ws[RADIX_BINS / 32], ss[RADIX_BINS], sl[RADIX_BINS], gs[RADIX_BINS + 1];
    __shared__ uint32_t wu[RADIX_BINS / 32], wr[RADIX_BINS / 32], gi[RADIX_BINS], goff[RADIX_BINS], groups, at, most;
    const int tid = threadIdx.x;
    if (tid == 0) most = 0;
    __syncthreads();
    if (tid < RADIX_BINS) {
        const uint32_t m = __reduce_max_sync(0xFFFFFFFFu, h <= (S)W ? (uint32_t)h : 0u);
        if ((tid & 31) == 0) atomicMax(&most, m);
    }
    const S s = radix_bin_scan<S>(tid < RADIX_BINS ? h : (S)0, ws);
    if (tid < RADIX_BINS) {
        row[tid] = s;
        ss[tid] = s;
        sl[tid] = h;
    }
    __syncthreads();
    const uint64_t parts = (q.slen + (CAP - most) - 1) / (CAP - most);
    const S part = (S)((q.slen + parts - 1) / parts);
    uint32_t b = 0;
    if (tid < RADIX_BINS)
        b = tid == 0 || h > (S)W || sl[tid - 1] > (S)W || s / part != ss[tid - 1] / part ? 1u : 0u;
    const uint32_t g = radix_bin_scan<uint32_t>(b, wu);
    if (tid < RADIX_BINS && b) {
        gs[g] = s;
        gi[g] = (uint32_t)tid;
    }
    if (tid == RADIX_BINS - 1) {
        groups = g + b;
        gs[g + b] = (S)q.slen;
    }
    __syncthreads();
    uint32_t nrec = 0;
    uint64_t len = 0, flags = 0;
    bool pure = false;
    if (tid < (int)groups) {
        len = (uint64_t)(gs[tid + 1] - gs[tid]);
        if (len > (uint64_t)CAP) {
            pure = map.pure(gi[tid]);
            if (pure)
                nrec = to.stay ? 0u : (uint32_t)((len + CAP - 1) / CAP);
            else if (to.next)
                to.next[atomicAdd(to.next_count, 1u)] = SbSeg{q.sbase + (uint64_t)gs[tid], len};
            else {
                nrec = 1;
                flags = SbRec::SLOW;
            }
        } else {
            nrec = len ? 1u : 0u;
        }
    }
    const uint32_t o = radix_bin_scan<uint32_t>(nrec, wr);
    if (tid == RADIX_BINS - 1) at = atomicAdd(to.rec_count, o + nrec);
    if (tid < RADIX_BINS) goff[tid] = pure ? o : 0xFFFFFFFFu;
    __syncthreads();
    if (nrec && !pure) {
        to.recs[at + o] = SbRec{q.sbase + (uint64_t)gs[tid], len | flags | to.flags};
        if (flags & SbRec::SLOW) to.slow[atomicAdd(to.slow_count, 1u)] = at + o;
    }
    // equal keys that have to move: pieces, by the whole CTA
    if (__syncthreads_or(pure && nrec)) {
        for (uint32_t k = 0; k < groups; ++k) {
            if (goff[k] == 0xFFFFFFFFu) continue;
            const uint64_t p0 = (uint64_t)gs[k], pl = (uint64_t)(gs[k + 1] - gs[k]);
            for (uint64_t i = tid; i * CAP < pl; i += NT) {
                const uint64_t rest = pl - i * CAP;
                to.recs[at + goff[k] + i] =
                    SbRec{q.sbase + p0 + i * CAP, (rest < (uint64_t)CAP ? rest : (uint64_t)CAP) | to.flags};
            }
        }
    }
    __syncthreads();
}

// Counts the level's slices: hist[segment][256]. The lanes of a warp spread over
// COPIES copies of the counters; a CTA takes a contiguous range of tiles and
// flushes its counters when the segment changes. Keys arrive by bulk copy, the
// next tile while this one is counted (segments start at any item: the stage
// takes the 16-byte chunks that enclose the tile); pairs are read directly. The
// CTA that completes a segment (a ticket counts its tiles) turns the counts into
// starts and hands the slices on. look (pairs): the look-back words of the pass,
// cleared here.
template <class T, class S>
__global__ void __launch_bounds__(512)
    sb_hist_kernel(SbBuffers<T> buf, int level, const SbTile* tiles, const uint32_t* tile_count,
                   const SbMap<typename Traits<T>::Key>* maps, const typename Traits<T>::Key* splitters, uint64_t xmask,
                   S* hist, uint32_t* done, SbHandOn to, S* look, int* err, uint32_t spin) {
    using Sh = SegBucketShape<T>;
    using K = typename Traits<T>::Key;
    constexpr int NT = 512, COPIES = 16, TILE = Sh::TILE, V = Vec<T>::N, STEPS = TILE / V / NT;
    static_assert(STEPS * V * NT == TILE, "whole vector steps");
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ uint32_t cnt[RADIX_BINS * COPIES];
    __shared__ K sp[SB_SPLITTERS + 1];
    __shared__ bool last;
    __shared__ __align__(8) uint64_t bar[2];
    const int tid = threadIdx.x, col = tid & (COPIES - 1);
    if (!Sh::STABLE && tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        mbar_init_fence();
    }
    grid_dep_wait();
    const uint32_t total = count_load(tile_count);
    const uint32_t t0 = (uint32_t)((uint64_t)total * blockIdx.x / gridDim.x);
    const uint32_t t1 = (uint32_t)((uint64_t)total * (blockIdx.x + 1) / gridDim.x);
    if (t0 >= t1) return;
    const bool from_tmp = buf.from_tmp(level);
    const T* in = from_tmp ? buf.tmp : buf.d;
    to.flags = from_tmp ? 0 : SbRec::TMP;
    to.stay = to.stay && from_tmp != buf.want_tmp;
    for (int i = tid; i < RADIX_BINS * COPIES; i += NT) cnt[i] = 0;
    SbDigit<T> dig;
    dig.xmask = xmask;
    dig.sp = sp;
    auto flush = [&](const SbTile& q, uint32_t flushed) {
        S* row = hist + (size_t)q.seg * RADIX_BINS;
        __syncthreads();
        if (tid < RADIX_BINS) {
            uint32_t s = 0;
#pragma unroll
            for (int c = 0; c < COPIES; ++c) {
                s += cnt[tid * COPIES + c];
                cnt[tid * COPIES + c] = 0;
            }
            if (s) {
                if constexpr (sizeof(S) == 8)
                    atomicAdd(reinterpret_cast<unsigned long long*>(row) + tid, (unsigned long long)s);
                else
                    atomicAdd(row + tid, s);
            }
        }
        __threadfence();
        __syncthreads();
        if (tid == 0) {
            const uint32_t nt = (uint32_t)((q.slen + TILE - 1) / TILE);
            last = atomicAdd(done + q.seg, flushed) + flushed == nt;
        }
        __syncthreads();
        if (last) {
            __threadfence();
            S h = 0;
            if (tid < RADIX_BINS) h = *(volatile S*)(row + tid);
            sb_hand_on<T, S, NT>(q, h, dig.map, row, to);
        }
    };
    // thread 0: a tile on its way into a stage
    auto issue = [&](const SbTile& r, uint32_t slot) {
        const int lead = (int)(r.base % V), nv = (lead + (int)r.cnt + V - 1) / V;
        mbar_arrive_expect(&bar[slot], (uint32_t)nv * 16u);
        bulk_load(smem_raw + slot * Sh::STAGE_BYTES, in + (r.base - lead), (uint32_t)nv * 16u, &bar[slot]);
    };
    SbTile q = tiles[t0], r = q;
    if constexpr (!Sh::STABLE) {
        if (tid == 0) issue(q, 0);
        __syncthreads();  // the barriers are set up
    }
    uint32_t since = t0;
    for (uint32_t t = t0;; ) {
        if (t + 1 < t1) r = tiles[t + 1];
        if (t == since) {  // first tile of a segment here
            dig.map = maps[q.seg];
            if (dig.map.mode == SB_SEARCH && tid <= SB_SPLITTERS)
                sp[tid] = splitters[(size_t)q.seg * (SB_SPLITTERS + 1) + tid];
            if (Sh::STABLE) __syncthreads();
        }
        const T* p = in + q.base;
        if constexpr (!Sh::STABLE) {
            const uint32_t slot = (t - t0) & 1u, parity = ((t - t0) >> 1) & 1u;
            const bool ok = mbar_wait(&bar[slot], parity, spin);
            // every thread is done with the other stage too
            if (__syncthreads_or(!ok)) {
                if (tid == 0) bulk_drain<2>(err, bar, 1u << slot, parity << slot);
                return;
            }
            if (tid == 0 && t + 1 < t1) issue(r, slot ^ 1u);
            p = reinterpret_cast<const T*>(smem_raw + slot * Sh::STAGE_BYTES) + q.base % V;
        }
        const bool vec = ((uintptr_t)p & 15) == 0 && q.cnt == TILE;
        dig.with_mode([&](auto mode) {
            constexpr uint32_t MODE = decltype(mode)::value;
            if (MODE == SB_LINEAR && vec) {
                uint4 x[STEPS];
#pragma unroll
                for (int j = 0; j < STEPS; ++j) x[j] = reinterpret_cast<const uint4*>(p)[j * NT + tid];
#pragma unroll
                for (int j = 0; j < STEPS; ++j) {
                    const T* e = reinterpret_cast<const T*>(&x[j]);
#pragma unroll
                    for (int k = 0; k < V; ++k) atomicAdd(&cnt[dig.template by<MODE>(e[k]) * COPIES + col], 1u);
                }
            } else {
#pragma unroll 8
                for (uint32_t i = tid; i < q.cnt; i += NT) atomicAdd(&cnt[dig.template by<MODE>(p[i]) * COPIES + col], 1u);
            }
        });
        if (look)
            for (int i = tid; i < RADIX_BINS; i += NT) look[(size_t)t * RADIX_BINS + i] = 0;
        ++t;
        if (t == t1) {
            flush(q, t - since);
            break;
        }
        if (r.seg != q.seg) {
            flush(q, t - since);
            since = t;
        }
        q = r;
    }
}

// ------------------------------------------------------------------- pass ---
// One partition level of keys-only items: count the tile's digits, claim each
// digit's output range, place the items in digit order in shared memory, write
// them out run by run. Per 32 keys the shared-memory pipe takes three random accesses of 3.5
// bank conflicts (count, place, store). Atomics of lanes with one digit would be
// serialised (31 cycles): a segment with a heavy key lets one lane count and
// place for all lanes that hold it, and a tile whose neighbours share digits
// (sorted or nearly sorted input: a warp's first step is uniform) does so where a
// step is uniform.
//
// LOOP: a resident grid for a level that is rarely needed; else one CTA per tile
// (a loop costs registers, and so resident warps).
template <class T, class S, bool LOOP>
__global__ void __launch_bounds__(SegBucketCfg<T>::NT, SegBucketCfg<T>::MINB)
    sb_pass_kernel(SbBuffers<T> buf, int level, const SbTile* tiles, const uint32_t* tile_count,
                   const SbMap<typename Traits<T>::Key>* maps, const typename Traits<T>::Key* splitters, uint64_t xmask,
                   S* cursor, const int* err) {
    using Sh = SegBucketShape<T>;
    using K = typename Traits<T>::Key;
    constexpr int NT = Sh::C::NT, IPT = Sh::C::IPT, TILE = Sh::TILE;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* skeys = reinterpret_cast<T*>(smem_raw);
    __shared__ uint32_t tab[RADIX_BINS], ws[RADIX_BINS / 32];
    __shared__ S goff[RADIX_BINS];
    __shared__ K sp[SB_SPLITTERS + 1];
    static_assert(NT >= RADIX_BINS && IPT % 4 == 0, "one thread per slice; four digits to a register");
    const int tid = threadIdx.x, lane = tid & 31;
    grid_dep_wait();
    uint32_t t = blockIdx.x;
    SbTile q = tiles[t];  // (the list has room for the grid: one latency with the count)
    const uint32_t total = count_load(tile_count);
    if (t >= total || err_wait_set(err)) return;
    const bool from_tmp = buf.from_tmp(level);
    const T* src = from_tmp ? buf.tmp : buf.d;
    T* dst = from_tmp ? buf.d : buf.tmp;
    SbDigit<T> dig;
    dig.xmask = xmask;
    dig.sp = sp;
    do {
        const int cnt = (int)q.cnt, mine = cnt - tid;
        T v[IPT];
        uint32_t dp[IPT / 4];  // the items' digits
        const bool whole = cnt == TILE;
        {
            const T* p = src + q.base;
            if (whole) {
#pragma unroll
                for (int i = 0; i < IPT; ++i) v[i] = p[i * NT + tid];
            } else {
#pragma unroll
                for (int i = 0; i < IPT; ++i) v[i] = p[min(i * NT + tid, cnt - 1)];
            }
        }
        dig.map = maps[q.seg];
        if (tid < RADIX_BINS) tab[tid] = 0;
        if (dig.map.mode == SB_SEARCH && tid <= SB_SPLITTERS) sp[tid] = splitters[(size_t)q.seg * (SB_SPLITTERS + 1) + tid];
        __syncthreads();
        dig.with_mode([&](auto mode) {
            constexpr uint32_t MODE = decltype(mode)::value;
#pragma unroll
            for (int i = 0; i < IPT; i += 4)
                dp[i / 4] = dig.template by<MODE>(v[i]) | dig.template by<MODE>(v[i + 1]) << 8 |
                            dig.template by<MODE>(v[i + 2]) << 16 | dig.template by<MODE>(v[i + 3]) << 24;
        });
        auto digit = [&](int i) -> uint32_t { return __byte_perm(dp[i / 4], 0, 0x4440 | (i & 3)); };
        const bool plain = dig.map.mode == SB_LINEAR &&
                           !__all_sync(0xFFFFFFFFu, digit(0) == __shfl_sync(0xFFFFFFFFu, digit(0), 0));
        // the lanes that one lane counts and places for: those with the heavy key,
        // or all of them in a uniform step
        auto joint = [&](int i) -> unsigned {
            const uint32_t d = digit(i);
            const bool in = i * NT < mine;
            if (dig.map.mode == SB_HEAVY) return __ballot_sync(0xFFFFFFFFu, in && d == dig.map.heavy_slice);
            const uint32_t d0 = __shfl_sync(0xFFFFFFFFu, d, 0);
            return __all_sync(0xFFFFFFFFu, in && d == d0) ? 0xFFFFFFFFu : 0u;
        };
        if (plain) {
#pragma unroll
            for (int i = 0; i < IPT; ++i)
                if (i * NT < mine) atomicAdd(&tab[digit(i)], 1u);
        } else {
#pragma unroll
            for (int i = 0; i < IPT; ++i) {
                const unsigned m = joint(i);
                if ((m >> lane) & 1u) {
                    if (lane == __ffs(m) - 1) atomicAdd(&tab[digit(i)], (uint32_t)__popc(m));
                } else if (i * NT < mine) {
                    atomicAdd(&tab[digit(i)], 1u);
                }
            }
        }
        __syncthreads();
        const uint32_t c = tid < RADIX_BINS ? tab[tid] : 0u;
        S g = 0;
        if (c) {
            S* cu = cursor + (size_t)q.seg * RADIX_BINS + tid;
            if constexpr (sizeof(S) == 8)
                g = (S)atomicAdd(reinterpret_cast<unsigned long long*>(cu), (unsigned long long)c);
            else
                g = atomicAdd(cu, c);
        }
        const uint32_t start = radix_bin_scan<uint32_t>(c, ws);
        if (tid < RADIX_BINS) tab[tid] = start;
        __syncthreads();
        if (plain) {
#pragma unroll
            for (int i = 0; i < IPT; ++i)
                if (i * NT < mine) skeys[atomicAdd(&tab[digit(i)], 1u)] = v[i];
        } else {
#pragma unroll
            for (int i = 0; i < IPT; ++i) {
                const unsigned m = joint(i);
                const bool in = i * NT < mine;
                uint32_t r = 0;
                if (m && lane == __ffs(m) - 1) r = atomicAdd(&tab[digit(i)], (uint32_t)__popc(m));
                const uint32_t r0 = m ? __shfl_sync(0xFFFFFFFFu, r, __ffs(m) - 1) : 0u;
                if ((m >> lane) & 1u)
                    r = r0 + __popc(m & ((1u << lane) - 1u));
                else if (in)
                    r = atomicAdd(&tab[digit(i)], 1u);
                if (in) skeys[r] = v[i];
            }
        }
        if (tid < RADIX_BINS) goff[tid] = g - (S)start;
        __syncthreads();
        // (o < slen always holds while the input does not change under the sort)
        T* out = dst + q.sbase;
        dig.with_mode([&](auto mode) {
            constexpr uint32_t MODE = decltype(mode)::value;
            if (MODE == SB_LINEAR && whole) {
#pragma unroll 8
                for (int i = 0; i < IPT; ++i) {
                    const T x = skeys[i * NT + tid];
                    const S o = goff[dig.template by<MODE>(x)] + (S)(i * NT + tid);
                    if (o < (S)q.slen) out[o] = x;
                }
            } else {
                for (int j = tid; j < cnt; j += NT) {
                    const T x = skeys[j];
                    const S o = goff[dig.template by<MODE>(x)] + (S)j;
                    if (o < (S)q.slen) out[o] = x;
                }
            }
        });
        if (!LOOP || (t += gridDim.x) >= total) break;
        q = tiles[t];
        __syncthreads();
    } while (true);
}

// ------------------------------------------------------------ stable pass ---
// One partition level that keeps the order of equal digits (single-pass scheme
// with decoupled look-back: Merrill and Garland 2016, Adinets and Merrill 2022).
// A CTA claims a tile, holds its items in registers, counts their digits (every
// 16 lanes against 256 words of their own), publishes the tile's counts, places
// the items in digit order in shared memory, and learns where each digit's items
// go by looking back over the counts of the tiles before it in the segment until
// it meets one that already knows its prefix. The segment's first tile starts
// from the slice starts. Tiles are claimed in order, so the tiles a look-back
// waits for are always held by running CTAs; a tile is claimed only once its CTA
// has finished the one before (claimed earlier, it held up everyone behind it:
// passes 2 to 3 times longer).
//
// Ranking. A word holds the next place of a digit (upper half) and, during a
// step, which of the 16 lanes have it (lower half): one shared-memory OR, one
// load, a population count, one store by the digit's last lane: 8 cycles per
// warp step and SM. Ballots over the eight bits take 13 to 26, match.any 61.
//
// A wait that expires (`spin` polls) records ERR_WAIT_EXPIRED; waiting CTAs see
// the word and stop, later passes return at once.
template <class T, class S>
__global__ void __launch_bounds__(SegBucketCfg<T>::NT, SegBucketCfg<T>::MINB)
    sb_stable_pass_kernel(SbBuffers<T> buf, int level, const SbTile* tiles, const uint32_t* tile_count,
                          const SbMap<typename Traits<T>::Key>* maps, const typename Traits<T>::Key* splitters,
                          uint64_t xmask, const S* start, S* look, unsigned* claim, int* err, uint32_t spin) {
    using Sh = SegBucketShape<T>;
    using W = LookWord<S>;
    using K = typename Traits<T>::Key;
    constexpr int NT = Sh::C::NT, IPT = Sh::C::IPT, NG = Sh::GROUPS, TILE = Sh::TILE;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* skeys = reinterpret_cast<T*>(smem_raw);
    uint32_t* table = reinterpret_cast<uint32_t*>(smem_raw + Sh::TILE_BYTES);  // [NG][256]
    __shared__ S goff[RADIX_BINS];
    __shared__ uint32_t ws[RADIX_BINS / 32];
    __shared__ K sp[SB_SPLITTERS + 1];
    __shared__ uint32_t next_tile;
    static_assert(NT == RADIX_BINS, "one thread per slice");
    const int tid = threadIdx.x, hl = tid & 15, grp = tid >> 4;
    uint32_t* gt = table + grp * RADIX_BINS;
    const unsigned one = 1u << hl, lt = one - 1u;
    grid_dep_wait();
    const uint32_t total_tiles = count_load(tile_count);
    if (total_tiles == 0) return;
    const bool from_tmp = buf.from_tmp(level);
    const T* src = from_tmp ? buf.tmp : buf.d;
    T* dst = from_tmp ? buf.d : buf.tmp;
    if (tid == 0) next_tile = atomicAdd(claim, 1u);
    if (__syncthreads_or(tid == 0 && err_wait_set(err))) return;
    SbDigit<T> dig;
    dig.xmask = xmask;
    dig.sp = sp;
    for (uint32_t t = next_tile; t < total_tiles; t = next_tile) {
        const SbTile q = tiles[t];
        const uint32_t ti = (uint32_t)((q.base - q.sbase) / TILE);  // the tile's number in its segment
        dig.map = maps[q.seg];
        if (dig.map.mode == SB_SEARCH) {
            if (tid <= SB_SPLITTERS) sp[tid] = splitters[(size_t)q.seg * (SB_SPLITTERS + 1) + tid];
            __syncthreads();
        }
        const int cnt = (int)q.cnt;
        T v[IPT];
        const int i0 = grp * (16 * IPT) + hl;
        const int mine = cnt - i0;  // item i of this thread exists when i * 16 < mine
        {
            const T* p = src + q.base;
            if (cnt == TILE) {
#pragma unroll
                for (int i = 0; i < IPT; ++i) v[i] = p[i0 + i * 16];
            } else {
#pragma unroll
                for (int i = 0; i < IPT; ++i) v[i] = p[min(i0 + i * 16, cnt - 1)];
            }
        }
        {
            uint4* z = reinterpret_cast<uint4*>(gt);
#pragma unroll
            for (int i = 0; i < RADIX_BINS / 64; ++i) z[i * 16 + hl] = make_uint4(0, 0, 0, 0);
        }
        __syncwarp();
        // the items' digits, and the group's counts (upper half of its words)
        uint32_t dp[(IPT + 3) / 4];
        dig.with_mode([&](auto mode) {
            constexpr uint32_t MODE = decltype(mode)::value;
#pragma unroll
            for (int i = 0; i < IPT; i += 4)
                dp[i / 4] = dig.template by<MODE>(v[i]) | dig.template by<MODE>(v[i + 1]) << 8 |
                            dig.template by<MODE>(v[i + 2]) << 16 | dig.template by<MODE>(v[i + 3]) << 24;
        });
        static_assert(IPT % 4 == 0, "four digits to a register");
        auto digit = [&](int i) -> uint32_t { return __byte_perm(dp[i / 4], 0, 0x4440 | (i & 3)); };
#pragma unroll
        for (int i = 0; i < IPT; ++i)
            if (i * 16 < mine) atomicAdd(&gt[digit(i)], 1u << 16);
        __syncthreads();
        // per bin: the tile's count, published, and the groups' first places
        uint32_t total = 0;
        S* my = look + (size_t)t * RADIX_BINS + tid;
#pragma unroll
        for (int g = 0; g < NG; ++g) total += table[g * RADIX_BINS + tid] >> 16;
        if (ti) look_store(my, W::COUNT | (S)total);
        const uint32_t first = radix_bin_scan<uint32_t>(total, ws);
        {
            uint32_t run = first;
#pragma unroll
            for (int g = 0; g < NG; ++g) {
                const uint32_t c = table[g * RADIX_BINS + tid] >> 16;
                table[g * RADIX_BINS + tid] = run << 16;
                run += c;
            }
        }
        __syncthreads();
        // rank and order the tile by digit in shared memory
#pragma unroll
        for (int i = 0; i < IPT; ++i) {
            const unsigned d = digit(i);
            const bool in = i * 16 < mine;
            if (in) atomicOr(&gt[d], one);
            __syncwarp();
            const uint32_t w = gt[d], m = w & 0xFFFFu;
            const uint32_t r = (w >> 16) + __popc(m & lt);
            __syncwarp();
            if (in && (m >> hl) == 1u) gt[d] = (r + 1) << 16;  // the digit's last lane
            __syncwarp();
            if (in) skeys[r] = v[i];
        }
        // where this tile's items of bin `tid` go inside the segment
        S excl = 0;
        bool ok = true;
        if (ti == 0) {
            excl = start[(size_t)q.seg * RADIX_BINS + tid];
        } else {
            constexpr int LB = 4;
            const S* p = my - RADIX_BINS;
            int left = (int)ti;  // tiles before this one in the segment
            uint32_t polls = 0;
            bool found = false;
            while (!found) {
                if (polls >= spin) {
                    ok = false;
                    break;
                }
                S s[LB];
#pragma unroll
                for (int k = 0; k < LB; ++k) s[k] = k < left ? look_load(p - (ptrdiff_t)k * RADIX_BINS) : (S)0;
                int used = 0;
#pragma unroll
                for (int k = 0; k < LB; ++k) {
                    if (used == k && !found && s[k]) {
                        excl += s[k] & W::MASK;
                        found = (s[k] & W::PREFIX) != 0;
                        ++used;
                    }
                }
                p -= (ptrdiff_t)used * RADIX_BINS;
                left -= used;
                if (!used) {
                    ++polls;
                    if ((polls & 63u) == 0 && err_wait_set(err)) {
                        ok = false;
                        break;
                    }
                }
            }
        }
        if (ok) look_store(my, W::PREFIX | (excl + (S)total));
        goff[tid] = excl - (S)first;
        if (__syncthreads_or(!ok)) {
            if (tid == 0) {
                atomicCAS(err, 0, ERR_WAIT_EXPIRED);
                atomicCAS(err, ERR_BAD_RUNS, ERR_WAIT_EXPIRED);
            }
            return;
        }
        if (tid == 0) next_tile = atomicAdd(claim, 1u);
        T* out = dst + q.sbase;
        // (o < slen always holds while the input does not change under the sort)
        dig.with_mode([&](auto mode) {
            constexpr uint32_t MODE = decltype(mode)::value;
#pragma unroll 4
            for (int i = 0; i < IPT; ++i) {
                const int j = i * NT + tid;
                if (j < cnt) {
                    const T x = skeys[j];
                    const S o = goff[dig.template by<MODE>(x)] + (S)j;
                    if (o < (S)q.slen) out[o] = x;
                }
            }
        });
        __syncthreads();
    }
}

// ------------------------------------------------------------ bucket sort ---
// One step of a stable byte pass, as radix_pass_kernel ranks: every 16 lanes
// own a stretch of items and 256 words of `table`; the words hold the items' next
// places when it returns from sb_byte_count (which gives thread b < 256 the count
// of digit b), and sb_byte_place calls put(place, i) for every item i.
template <class T, int NT, int IPT, class Digit>
__device__ __forceinline__ uint32_t sb_byte_count(uint32_t* table, uint32_t* ws, int mine, Digit digit) {
    constexpr int NG = NT / 16;
    const int tid = threadIdx.x, hl = tid & 15;
    uint32_t* gt = table + (tid >> 4) * RADIX_BINS;
    uint4* z = reinterpret_cast<uint4*>(gt);
#pragma unroll
    for (int i = 0; i < RADIX_BINS / 64; ++i) z[i * 16 + hl] = make_uint4(0, 0, 0, 0);
    __syncwarp();
#pragma unroll
    for (int i = 0; i < IPT; ++i)
        if (i * 16 < mine) atomicAdd(&gt[digit(i)], 1u << 16);
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
    return total;
}
template <int IPT, class Digit, class Put>
__device__ __forceinline__ void sb_byte_place(uint32_t* table, int mine, Digit digit, Put put) {
    const int hl = threadIdx.x & 15;
    uint32_t* gt = table + (threadIdx.x >> 4) * RADIX_BINS;
    const unsigned one = 1u << hl, lt = one - 1u;
#pragma unroll
    for (int i = 0; i < IPT; ++i) {
        const bool in = i * 16 < mine;
        const unsigned d = in ? digit(i) : 0;
        if (in) atomicOr(&gt[d], one);
        __syncwarp();
        const uint32_t x = gt[d], m = x & 0xFFFFu;
        const uint32_t r = (x >> 16) + __popc(m & lt);
        __syncwarp();
        if (in && (m >> hl) == 1u) gt[d] = (r + 1) << 16;
        __syncwarp();
        if (in) put(r, d, i);
    }
}

// A slice that does not fit: stable byte passes by one CTA in global memory, between
// its place in either buffer (a: where it is). Bytes that all keys share are skipped.
// (Not inlined: its registers are not the other buckets'.)
template <class T>
__device__ __noinline__ void sb_sort_long(T* a, T* b, T* want, uint64_t len, uint64_t xin, uint64_t xout) {
    unsigned char* smem_raw = bk_smem();
    using Sh = BucketShape<T>;
    using K = typename Traits<T>::Key;
    using Count = unsigned long long;
    constexpr int NT = Sh::C::S_NT, IPT = Sh::C::S_IPT;
    // where a bucket's items stand otherwise (static shared memory would count for every bucket)
    Count* cnt = reinterpret_cast<Count*>(smem_raw);
    Count *place = cnt + RADIX_BINS, *ws8 = place + RADIX_BINS;
    uint32_t* ws = reinterpret_cast<uint32_t*>(ws8 + RADIX_BINS / 32);
    uint32_t* table = reinterpret_cast<uint32_t*>(smem_raw + Sh::KEYS_BYTES);
    static_assert(Sh::KEYS_BYTES >= (2 * RADIX_BINS + RADIX_BINS / 32) * 8 + RADIX_BINS / 32 * 4, "they fit");
    const int tid = threadIdx.x, i0 = (tid >> 4) * (16 * IPT) + (tid & 15);
    T w[IPT];
#pragma unroll 1
    for (int byte = 0; byte < (int)sizeof(K); ++byte) {
        auto digit_of = [&](const T& v) -> unsigned {
            return (unsigned)(Traits<T>::key(bk_flip(v, xin)) >> (8 * byte)) & 255u;
        };
        auto digit = [&](int i) -> unsigned { return digit_of(w[i]); };
        if (tid < RADIX_BINS) cnt[tid] = 0;
        __syncthreads();
        for (uint64_t i = tid; i < len; i += NT) atomicAdd(&cnt[digit_of(a[i])], (Count)1);
        __syncthreads();
        const Count c = tid < RADIX_BINS ? cnt[tid] : 0;
        if (__syncthreads_or(c == (Count)len)) continue;
        const Count p0 = radix_bin_scan<Count>(c, ws8);
        if (tid < RADIX_BINS) place[tid] = p0;
        __syncthreads();
        for (uint64_t t = 0; t < len; t += (uint64_t)NT * IPT) {
            const int have = (int)(len - t < (uint64_t)NT * IPT ? len - t : (uint64_t)NT * IPT), mine = have - i0;
#pragma unroll
            for (int i = 0; i < IPT; ++i)
                if (i * 16 < mine) w[i] = a[t + i0 + i * 16];
            const uint32_t n = sb_byte_count<T, NT, IPT>(table, ws, mine, digit);
            // places in the tile become places in the bucket: cnt holds the
            // digit's place minus its start in the tile, modulo 2^64
            const uint32_t start = radix_bin_scan<uint32_t>(n, ws);
            if (tid < RADIX_BINS) cnt[tid] = place[tid] - start;
            __syncthreads();
            sb_byte_place<IPT>(table, mine, digit, [&](uint32_t o, unsigned dg, int i) {
                const Count p = cnt[dg] + o;
                if (p < len) b[p] = w[i];
            });
            __syncthreads();
            if (tid < RADIX_BINS) place[tid] += n;
            __syncthreads();
        }
        T* x = a;
        a = b;
        b = x;
    }
    if (a != want || xin != xout)
        for (uint64_t i = tid; i < len; i += NT) want[i] = bk_flip(a[i], xin ^ xout);
}

// The buckets of a plain bucket sort that did not give up: [start[b], start[b + 1]) of d
// or tmp.
struct SbStarts {
    const uint32_t* start;
    uint32_t buckets;
    bool in_tmp;
};

// Sorts every bucket, one CTA each (bk_sort_bucket; a loop over buckets costs registers,
// 2^28 uint32 keys 1.67 ms instead of 1.24): those of the list, or the plain bucket
// sort's, so that no launch is for buckets of the other kind only (2 ns for every CTA
// that finds nothing to do). The CTAs from `first` on take the rest of the list in turn:
// the few buckets beyond the grid, and slices that did not fit.
// LOOP (32-bit keys behind a plain bucket sort, whose last kernel is one of its own):
// resident CTAs take all of the list in turn, so that few find nothing to do in the usual
// case (one CTA a bucket would cost 2^28 keys 0.2 ms there). The loop's variable stands in
// shared memory.
template <class T, bool LOOP>
__global__ void __launch_bounds__(BucketCfg<T>::S_NT, BucketCfg<T>::S_MINB)
    sb_sort_kernel(SbBuffers<T> buf, SbStarts plain, const SbRec* recs, const uint32_t* slow, const SbCounts* cn,
                   uint32_t first, uint64_t xin, uint64_t xout) {
    if constexpr (LOOP) {
        __shared__ volatile uint32_t next;
        if (threadIdx.x == 0) next = blockIdx.x;
        grid_dep_wait();
#pragma unroll 1
        while (true) {
            __syncthreads();
            const uint32_t at = next;
            if (at >= count_load(&cn->recs)) return;
            const SbRec r = recs[at];
            const bool moved = (r.what & SbRec::TMP) != 0;
            T *a = (moved ? buf.tmp : buf.d) + r.base, *out = buf.want() + r.base;
            if (r.what & SbRec::SLOW) {
                sb_sort_long<T>(a, (moved ? buf.d : buf.tmp) + r.base, out, r.what & SbRec::LEN, xin, xout);
            } else {
                const int cnt = (int)(r.what & SbRec::LEN);
                bk_sort_init<T>();
                if (!bk_sort_bucket<T, BK_LEAVE>(a, out, cnt, xin, xout)) bk_sort_left<T>(a, out, cnt, xin, xout);
            }
            __syncthreads();
            if (threadIdx.x == 0) next = next + gridDim.x;
        }
    }
    bk_sort_init<T>();
    grid_dep_wait();
    const uint32_t at = blockIdx.x;
    const T* src;
    uint64_t base;
    int cnt;
    // (32-bit keys: the plain bucket sort has a last kernel of its own)
    if (sizeof(typename Traits<T>::Key) == 8 && plain.start && route_load(buf.route) == ROUTE_BUCKETS) {
        if (at >= plain.buckets) return;
        const uint32_t b0 = plain.start[at], b1 = plain.start[at + 1];
        if (b1 <= b0 || b1 - b0 > (uint32_t)BucketShape<T>::CAP) return;
        src = plain.in_tmp ? buf.tmp : buf.d;
        base = b0;
        cnt = (int)(b1 - b0);
    } else if (at < first) {
        const SbRec r = recs[at];  // (the list has room for the grid: one latency with the count)
        if (at >= count_load(&cn->recs) || (r.what & SbRec::SLOW)) return;
        src = (r.what & SbRec::TMP) ? buf.tmp : buf.d;
        base = r.base;
        cnt = (int)(r.what & SbRec::LEN);
    } else {
        const uint32_t left = count_load(&cn->slow), all = count_load(&cn->recs);
        const uint32_t total = left + (all > first ? all - first : 0u);
        for (uint32_t h = at - first; h < total; h += gridDim.x - first) {
            const SbRec r = recs[h < left ? slow[h] : first + (h - left)];
            if (h >= left && (r.what & SbRec::SLOW)) continue;  // (once, by its place in `slow`)
            const uint64_t len = r.what & SbRec::LEN;
            const bool moved = (r.what & SbRec::TMP) != 0;
            T *a = (moved ? buf.tmp : buf.d) + r.base, *b = (moved ? buf.d : buf.tmp) + r.base;
            if (len > (uint64_t)BucketShape<T>::CAP)
                sb_sort_long<T>(a, b, buf.want() + r.base, len, xin, xout);
            else
                bk_sort_settled<T>(a, buf.want() + r.base, (int)len, xin, xout);
            __syncthreads();
        }
        return;
    }
    src += base;
    T* const out = buf.want() + base;
    if (!bk_sort_bucket<T, BK_LEAVE>(src, out, cnt, xin, xout)) bk_sort_left<T>(src, out, cnt, xin, xout);
}

}  // namespace origami
