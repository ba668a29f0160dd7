// Host launchers of the bucket sort (buckets.cuh) and of what stands behind it: the
// radix passes (radix.cuh) for 32-bit keys, the levels of the segmented bucket sort
// (seg_buckets.cuh) for 64-bit keys.
#pragma once
#include <algorithm>
#include <string>

#include "buckets.cuh"
#include "dispatch.h"
#include "pipeline.cuh"
#include "profiler.h"
#include "radix.cuh"
#include "seg_bucket_host.cuh"

namespace origami {

constexpr uint64_t RADIX_LEAST = 1 << 14;
constexpr uint64_t BK_MOST = 1ull << 31;  // items of a bucket sort: fewer

// Segments of a radix sort: the whole array, or chunks of sort_n items.
template <class T>
struct RadixPlan {
    using Sh = RadixShape<T>;
    uint64_t n, len;     // items; items per segment
    uint64_t tiles, nseg;
    uint32_t shift;      // log2(tiles per segment); 31: one segment
    bool wide;           // segments of 2^30 items or more: 64-bit look-back words
    RadixPlan(uint64_t n_, uint64_t sort_n) : n(n_), len(chunk_limit(n_, sort_n)) {
        tiles = (n + Sh::TILE - 1) / Sh::TILE;
        nseg = (n + len - 1) / len;
        shift = 31;
        if (nseg > 1)
            for (shift = 0; ((uint64_t)Sh::TILE << shift) < len;) ++shift;
        wide = len >= (1ull << 30);
    }
    // One bucket; else enough items for several launches (10,000 uint32 keys 27 us by
    // buckets, 26 by merges), whole tiles per segment, and tile numbers that fit 31 bits.
    // Not chunks of 2^31 uint32 keys in all and more, which the bucket sort does not take:
    // radix passes, 6.6 ms for 2^28 Zipf keys, have merges of 3.3 to 5.1 ms against them.
    static bool fits(uint64_t n, uint64_t sort_n) {
        const uint64_t len = chunk_limit(n, sort_n);
        if (sizeof(typename Traits<T>::Key) == 4 && len < n && n >= BK_MOST) return false;
        if (n < 2 || (len == n && n <= (uint64_t)BucketShape<T>::CAP)) return n >= 2;
        return n >= RADIX_LEAST && (len == n || len % Sh::TILE == 0) && n / Sh::TILE < (1ull << 31) - 2;
    }
};

// Bucket sort of a full sort or of chunks: bits per level, 0 when it does not
// take the call: more than 65,536 buckets of the mean size (2^LOG_TARGET: two thirds of
// what fits for uint32 keys, half for wider items), so sorts and chunks of 2^28 + 65,536
// uint32 keys, 2^27 + 65,536 wider items and more; or fewer than 16 buckets.
template <class T>
struct BucketPlan {
    using Sh = BucketShape<T>;
    int b1 = 0, b2 = 0;
    uint64_t tiles = 0, tiles2 = 0, nbuckets = 0;
    BucketPlan(const RadixPlan<T>& p) {
        if (p.n >= BK_MOST) return;
        int bits = 0;
        while ((p.len >> bits) > (1ull << Sh::C::LOG_TARGET)) ++bits;
        // short sorts: one level can have up to 256 buckets, enough for every SM
        while (bits < 8 && (p.nseg << bits) < RADIX_BINS && (p.len >> bits) > 256) ++bits;
        if (bits < 4 || bits > BK_MAX_BITS) return;
        if (p.nseg > 1 && (p.len % Sh::TILE != 0 || p.nseg > (1u << 20))) return;
        // two levels of about equal width: few slices would serialise the atomics
        b1 = bits > 8 ? (bits + 1) / 2 : bits;
        b2 = bits - b1;
        tiles = (p.n + Sh::TILE - 1) / Sh::TILE;
        tiles2 = b2 ? tiles + (p.nseg << b1) : 0;
        nbuckets = p.nseg << bits;
    }
    bool on() const { return b1 > 0; }
    // rows of counts where one read counts both levels (one segment): one for every SM,
    // and four tiles each
    uint32_t rows(const RadixPlan<T>& p) const {
        return b2 && p.nseg == 1 ? (uint32_t)std::min<uint64_t>(sm_count(), (tiles + 3) / 4) : 0u;
    }
};

// What stands behind the bucket sort, and sorts where it does not take the call.
//   64-bit keys: the levels. Radix passes would read the keys once more for every byte, the
// levels do for every 256 slices, whatever the width: 2^27 uint64 Zipf keys 8.0 ms by radix
// passes and 3.4 by levels, 2^26 pairs 5.1 and 3.3, normally distributed keys 7.6 and 4.0,
// 5.6 and 2.4.
//   uint32 keys, one segment: radix passes, four of them and fewer launches (2^20 Zipf keys
// 0.074 ms, by levels some 0.11; 2^28 6.5 and 4.9, which one more path would not be for).
//   uint32 keys in chunks: by merges chunks took the less the shorter they are, so radix
// passes lost up to 2.4 times there. 2^28 keys, ms, merges alone / radix passes, levels,
// merges behind the bucket sort:
//     chunks of      2^16                    2^17                    2^19
//     Zipf keys      2.9 / 6.9, 6.4, 4.2     3.3 / 6.7, 7.0, 4.2     4.0 / 6.7, 5.4, 5.1
//     log-uniform    2.9 / 6.6, 5.4, 3.9     3.3 / 6.6, 4.9, 4.2     4.0 / 6.6, 4.9, 5.0
//     one chunk Zipf 2.9 / 4.3, 3.9, 4.1     3.3 / 4.2, 3.7, 4.4     4.0 / 4.0, 3.5, 5.2
// Merges up to 2^17 keys a chunk (one 16-way pass after the tile sort: three launches), the
// levels up to 2^20 (from there on one crowded chunk costs them a partition: chunks of 2^21
// 4.1 by radix passes, 5.8) in sorts of 2^25 keys and more: their launches, two more than
// radix passes', cost 2^22 uniform keys 7 of 69 us.
enum class Behind { RADIX, LEVELS, MERGES };
constexpr uint64_t MERGES_CHUNK = 1 << 17, MERGES_FROM = 1 << 22, LEVELS_CHUNK = 1 << 20, LEVELS_FROM = 1 << 25;
constexpr int MERGES_CODE = 16;  // shape: 16-way
template <class T>
Behind behind(const RadixPlan<T>& p, const BucketPlan<T>& bk) {
    if (sizeof(typename Traits<T>::Key) == 8) return Behind::LEVELS;
    if (!bk.on() || p.nseg <= 1) return Behind::RADIX;
    if (p.len <= MERGES_CHUNK) return p.n >= MERGES_FROM ? Behind::MERGES : Behind::RADIX;
    return p.len <= LEVELS_CHUNK && p.n >= LEVELS_FROM ? Behind::LEVELS : Behind::RADIX;
}
template <class T>
SegBucketPlan<T> behind_plan(const RadixPlan<T>& p, const BucketPlan<T>& bk) {
    return SegBucketPlan<T>(p.n, bk.b2 ? p.nseg << bk.b1 : p.nseg, p.len);
}

// Device scratch of one sort (each part 256-byte aligned):
//   bucket sort: slice starts and cursors of both levels, slice maps, tiles of
//   the second level and their count
//   look 1/0   look-back words of the odd / even radix passes, or of the second /
//              first level of pairs, 256 per tile
//   hist 1/2   counts of the bucket sort's levels
//   hist       digit counts of the radix passes, [segment][digit][256]
//   words      the passes' tile counters, the bucket sort's route and tile count
//   tail       256 bytes: the error word; the counters of the levels behind
// From `zero` on everything starts at 0 (one memset). First of all the scratch of the
// levels or merges behind.
template <class T>
struct RadixScratch {
    using K = typename Traits<T>::Key;
    uint64_t bytes = 0, zero_bytes = 0;
    char* zero = nullptr;
    void* look[2] = {nullptr, nullptr};
    uint32_t *start1 = nullptr, *start2 = nullptr, *cursor1 = nullptr, *cursor2 = nullptr, *count2 = nullptr, *done = nullptr;
    SliceMap<K>* maps = nullptr;
    uint32_t* rows = nullptr;
    BkTile* tiles2 = nullptr;
    uint32_t *hist1 = nullptr, *hist2 = nullptr;
    void* hist = nullptr;
    int *err = nullptr, *route = nullptr;
    unsigned* claim = nullptr;
    RadixScratch(void* base, const RadixPlan<T>& p, const BucketPlan<T>& bk) {
        constexpr bool ST = BucketShape<T>::STABLE;
        const Behind rest = behind(p, bk);
        const bool passes = rest == Behind::RADIX;
        const uint64_t w = p.wide ? 8 : 4;
        char* b = static_cast<char*>(base);
        uint64_t o = 0;
        auto take = [&](uint64_t sz) {
            char* r = b ? b + o : nullptr;
            o += (sz + 255) & ~255ull;
            return r;
        };
        auto words = [&](uint64_t k) { return reinterpret_cast<uint32_t*>(take(k * 4)); };
        if (rest == Behind::LEVELS) o += SegBucketScratch<T>(nullptr, behind_plan(p, bk), nullptr, false).bytes;
        if (rest == Behind::MERGES) o += PipeScratch<T>(nullptr, p.n, p.len, MERGES_CODE, 0).bytes;
        if (bk.on()) {
            start1 = words((p.nseg << bk.b1) + 1);
            if (!ST) cursor1 = words(p.nseg << bk.b1);
            maps = reinterpret_cast<SliceMap<K>*>(take(p.nseg * sizeof(SliceMap<K>)));
            if (bk.b2) {
                start2 = words(bk.nbuckets + 1);
                if (!ST) cursor2 = words(bk.nbuckets);
                tiles2 = reinterpret_cast<BkTile*>(take(bk.tiles2 * sizeof(BkTile)));
                rows = words((uint64_t)bk.rows(p) << (bk.b1 + bk.b2 - 1));
            }
        }
        // the second level's words: the first pass clears those of its own tiles
        const bool look_pairs = ST && bk.on();
        if (look_pairs ? bk.b2 > 0 : passes) look[1] = take(std::max(p.tiles, ST ? bk.tiles2 : 0) * RADIX_BINS * w);
        uint64_t z = o;
        if (look_pairs && bk.b2) z -= (bk.tiles2 - bk.tiles) * RADIX_BINS * w;
        if (look_pairs || passes) look[0] = take(p.tiles * RADIX_BINS * w);
        if (!look_pairs) z = o;  // (cleared by radix_hist_kernel)
        if (bk.on()) {
            hist1 = words(p.nseg << bk.b1);
            if (bk.b2) hist2 = words(bk.nbuckets);
        }
        if (passes) hist = take(p.nseg * RadixShape<T>::DIGITS * RADIX_BINS * w);
        claim = words(16);
        err = reinterpret_cast<int*>(take(256));
        if (b) {
            route = reinterpret_cast<int*>(claim + 12);
            count2 = claim + 13;
            done = claim + 14;
            zero = b + z;
        }
        zero_bytes = o - z;
        bytes = o;
    }
};

template <class T>
uint64_t radix_scratch_bytes(uint64_t n, uint64_t sort_n) {
    const RadixPlan<T> p(n, sort_n);
    return RadixScratch<T>(nullptr, p, BucketPlan<T>(p)).bytes;
}

// The radix passes: d -> want (d or tmp). With `route` they stand behind a
// bucket sort and run only where it gave up.
template <class T, class S>
void radix_launch(T* d, T* tmp, T* want, const RadixPlan<T>& p, const RadixScratch<T>& sc, const int* route,
                  cudaStream_t st) {
    using Sh = RadixShape<T>;
    using G = RadixUniform;
    using D = ByteDigit<T, S>;
    // kernel attributes and grids, once per process
    static const uint32_t g_hist = resident_ctas((const void*)radix_hist_kernel<T, S, G>, 512, radix_hist_smem<T>());
    static const uint32_t g_pass = resident_ctas((const void*)radix_pass_kernel<T, S, G, D>, Sh::NT, Sh::SMEM);
    static const std::string n_hist = std::string("radix_hist<") + TypeName<T>::v + ">";
    static const std::string n_pass = std::string("radix_pass<") + TypeName<T>::v + ">";
    const uint32_t tiles = (uint32_t)p.tiles;
    const G geo{p.n, p.len, p.shift};
    S* hist = static_cast<S*>(sc.hist);
    launch(n_hist.c_str(), st, [&] {
        launch_dependent(radix_hist_kernel<T, S, G>, dim3(std::min(tiles, g_hist)), dim3(512), radix_hist_smem<T>(), st,
                         (const T*)d, (const T*)tmp, want, geo, tiles, hist, static_cast<S*>(sc.look[0]), route);
    });
    T* src = want;
    T* dst = want == d ? tmp : d;
    static_assert(Sh::DIGITS % 2 == 0, "the passes end in the buffer they start from");
    for (int b = 0; b < Sh::DIGITS; ++b) {
        launch(n_pass.c_str(), st, [&] {
            launch_dependent(radix_pass_kernel<T, S, G, D>, dim3(std::min(tiles, g_pass)), dim3(Sh::NT), Sh::SMEM, st,
                             (const T*)src, dst, geo, tiles, D(hist, b), static_cast<S*>(sc.look[b & 1]),
                             b + 1 < Sh::DIGITS ? static_cast<S*>(sc.look[(b + 1) & 1]) : (S*)nullptr, sc.claim + b,
                             sc.err, wait_limit(), route, false);
        });
        std::swap(src, dst);
    }
}

// The bucket sort: d -> want (d or tmp), *route set where it gives up.
template <class T>
void bucket_launch(T* d, T* tmp, T* want, const RadixPlan<T>& p, const BucketPlan<T>& bk, uint64_t xmask,
                   uint64_t xout, const RadixScratch<T>& sc, uint32_t nzero, cudaStream_t st) {
    using Sh = BucketShape<T>;
    using RSh = RadixShape<T>;
    using K = typename Traits<T>::Key;
    using G1 = RadixUniform;
    using G2 = BkListed;
    using D = SliceDigitStable<T>;
    constexpr bool ST = Sh::STABLE;
    constexpr size_t SAMPLE_SMEM = ((1u << BK_MAX_BITS) / 2 + 1) * 4;
    static const uint32_t g_hist = resident_ctas((const void*)bk_hist_kernel<T, G1>, 512, 0);
    static const uint32_t g_part = [] {
        cudaFuncSetAttribute(bk_sample_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SAMPLE_SMEM);
        if constexpr (sizeof(K) == 4)
            cudaFuncSetAttribute(bk_sort_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Sh::SORT_SMEM);
        if constexpr (ST) {
            resident_ctas((const void*)radix_pass_kernel<T, uint32_t, G2, D>, RSh::NT, RSh::SMEM);
            return resident_ctas((const void*)radix_pass_kernel<T, uint32_t, G1, D>, RSh::NT, RSh::SMEM);
        } else {
            cudaFuncSetAttribute(bk_pass_kernel<T, G1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Sh::PASS_SMEM);
            cudaFuncSetAttribute(bk_pass_kernel<T, G2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Sh::PASS_SMEM);
            return 0u;
        }
    }();
    static const std::string n_sample = std::string("bucket_sample<") + TypeName<T>::v + ">";
    static const std::string n_hist = std::string("bucket_hist<") + TypeName<T>::v + ">";
    static const std::string n_scan = std::string("bucket_scan<") + TypeName<T>::v + ">";
    static const std::string n_pass = std::string("bucket_pass<") + TypeName<T>::v + ">";
    static const std::string n_sort = std::string("bucket_sort<") + TypeName<T>::v + ">";
    const int bits = bk.b1 + bk.b2;
    const uint32_t nseg = (uint32_t)p.nseg, tiles = (uint32_t)bk.tiles, n32 = (uint32_t)p.n;
    // (the partition tile may differ from the radix passes')
    uint32_t shift = 31;
    if (nseg > 1)
        for (shift = 0; ((uint64_t)Sh::TILE << shift) < p.len;) ++shift;
    const G1 geo{p.n, p.len, shift};
    launch(n_sample.c_str(), st, [&] {
        bk_sample_kernel<T><<<nseg, 1024, ((1u << bits) / 2 + 1) * 4, st>>>(d, p.n, p.len, xmask, bk.b1, bk.b2,
                                                                            (uint64_t)Sh::CAP, sc.maps, sc.route,
                                                                            reinterpret_cast<uint4*>(sc.zero), nzero);
    });
    const uint32_t nrows = bk.rows(p);
    if (nrows) {
        static const std::string n_all = std::string("bucket_hist_all<") + TypeName<T>::v + ">";
        static const std::string n_sum = std::string("bucket_sum<") + TypeName<T>::v + ">";
        static const std::string n_list = std::string("bucket_list<") + TypeName<T>::v + ">";
        static const bool configured = [] {
            cudaFuncSetAttribute(bk_hist_all_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 << BK_MAX_BITS);
            return true;
        }();
        (void)configured;
        launch(n_all.c_str(), st, [&] {
            launch_dependent(bk_hist_all_kernel<T>, dim3(nrows), dim3(1024), (size_t)2 << bits, st, (const T*)d, p.n,
                             (const SliceMap<K>*)sc.maps, xmask, bits, sc.rows, sc.route);
        });
        launch(n_sum.c_str(), st, [&] {
            launch_dependent(bk_sum_kernel<T>, dim3(1u << bk.b1), dim3(256), 0, st, (const uint32_t*)sc.rows, nrows, bk.b1,
                             bk.b2, sc.hist1, sc.hist2, sc.route);
        });
        launch(n_list.c_str(), st, [&] {
            launch_dependent(bk_list_kernel<T>, dim3(1u << bk.b1), dim3(256), 0, st, p.n, bk.b1, bk.b2,
                             (const uint32_t*)sc.hist1, (const uint32_t*)sc.hist2, sc.start1, sc.cursor1, sc.start2,
                             sc.cursor2, sc.tiles2, sc.count2, (const int*)sc.route);
        });
    }
    auto level = [&](auto geo_l, const T* src, T* dst, uint32_t tiles_l, int shift_l, int bits_l, uint32_t map_shift,
                     uint32_t segs, const uint32_t* seg_start, uint32_t* hist, uint32_t* start, uint32_t* cursor,
                     bool last, int full_route, void* look, void* look_next, unsigned* claim) {
        using G = decltype(geo_l);
        const BkScan to{start, cursor, last ? (BkTile*)nullptr : sc.tiles2, sc.count2, sc.route, full_route, p.n, segs - 1};
        if (!nrows) launch(n_hist.c_str(), st, [&] {
            launch_dependent(bk_hist_kernel<T, G>, dim3(std::min(tiles_l, g_hist)), dim3(512), 0, st, src, geo_l, tiles_l,
                             (const SliceMap<K>*)sc.maps, map_shift, xmask, shift_l, bits_l, hist,
                             (const int*)sc.route, to, segs == 1 ? sc.done : (uint32_t*)nullptr);
        });
        if (!nrows && segs > 1) launch(n_scan.c_str(), st, [&] {
            launch_dependent(bk_scan_kernel<T>, dim3(segs), dim3(RADIX_BINS), 0, st, (const uint32_t*)hist, bits_l,
                             seg_start, p.len, to);
        });
        launch(n_pass.c_str(), st, [&] {
            if constexpr (ST) {
                D dig;
                dig.xmask = xmask;
                dig.shift = shift_l;
                dig.mask = (1u << bits_l) - 1;
                dig.maps = sc.maps;
                dig.map_shift = map_shift;
                dig.start = start;
                dig.bits = bits_l;
                launch_dependent(radix_pass_kernel<T, uint32_t, G, D>, dim3(std::min(tiles_l, g_part)), dim3(RSh::NT),
                                 RSh::SMEM, st, src, dst, geo_l, tiles_l, dig, static_cast<uint32_t*>(look),
                                 static_cast<uint32_t*>(look_next), claim, sc.err, wait_limit(), (const int*)sc.route,
                                 true);
            } else {
                launch_dependent(bk_pass_kernel<T, G>, dim3(tiles_l), dim3(Sh::C::NT), Sh::PASS_SMEM, st, src, dst, geo_l,
                                 tiles_l, (const SliceMap<K>*)sc.maps, map_shift, xmask, shift_l, bits_l, cursor, n32,
                                 (const int*)sc.route);
            }
        });
    };
    const T* cur = tmp;
    level(geo, d, tmp, tiles, bk.b2, bk.b1, 0u, nseg, (const uint32_t*)nullptr, sc.hist1, sc.start1, sc.cursor1, !bk.b2,
          (int)ROUTE_RADIX, sc.look[0], bk.b2 ? sc.look[1] : nullptr, sc.claim + 8);
    if (bk.b2) {
        level(G2{sc.tiles2, sc.count2}, tmp, d, (uint32_t)bk.tiles2, 0, bk.b2, (uint32_t)bk.b1, nseg << bk.b1,
              (const uint32_t*)sc.start1, sc.hist2, sc.start2, sc.cursor2, true, (int)ROUTE_RADIX_MOVED, sc.look[1],
              (void*)nullptr, sc.claim + 9);
        cur = d;
    }
    // (64-bit keys: the last kernel of the levels behind sorts these buckets too)
    if constexpr (sizeof(K) == 4) launch(n_sort.c_str(), st, [&] {
        launch_dependent(bk_sort_kernel<T>, dim3((unsigned)bk.nbuckets), dim3(Sh::C::S_NT), Sh::SORT_SMEM, st, cur, want,
                         (const uint32_t*)(bk.b2 ? sc.start2 : sc.start1), xmask, xout, n32, (const int*)sc.route);
    });
}

// A sort of one bucket: d -> want by one launch, without scratch or waits. err (or null)
// is cleared.
template <class T>
bool one_bucket(uint64_t n, uint64_t sort_n) {
    return n >= 2 && n <= (uint64_t)BucketShape<T>::CAP && chunk_limit(n, sort_n) == n;
}
template <class T>
cudaError_t bucket_one(const T* d, T* want, uint64_t n, uint64_t key_mask, uint64_t out_mask, int* err, cudaStream_t st) {
    using Sh = BucketShape<T>;
    static const std::string n_one = std::string("bucket_one<") + TypeName<T>::v + ">";
    static const bool configured = [] {
        cudaFuncSetAttribute(bk_one_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Sh::SORT_SMEM);
        return true;
    }();
    (void)configured;
    launch(n_one.c_str(), st, [&] {
        bk_one_kernel<T><<<1, Sh::C::S_NT, Sh::SORT_SMEM, st>>>(d, want, (int)n, key_mask, out_mask, err);
    });
    return cudaGetLastError();
}

// Sorts d[0..n) in chunks of sort_n (0 = one full sort) into `want` (d or tmp):
// by buckets where the geometry allows it, with radix passes or levels behind them
// for what does not spread; else by those. key_mask: the sign flip of keys
// read; out_mask: of keys written. `scratch` holds
// radix_scratch_bytes<T>(n, sort_n) bytes.
template <class T>
cudaError_t radix_sort(T* d, T* tmp, uint64_t n, uint64_t sort_n, uint64_t key_mask, uint64_t out_mask, T* want,
                       void* scratch, cudaStream_t st) {
    const RadixPlan<T> p(n, sort_n);
    const BucketPlan<T> bk(p);
    const RadixScratch<T> sc(scratch, p, bk);
    if (one_bucket<T>(n, sort_n)) return bucket_one<T>(d, want, n, key_mask, out_mask, sc.err, st);
    // one segment's sample kernel clears what is not much by itself (2^20 uint32 keys: a
    // memset takes 2 us)
    const bool self = bk.on() && p.nseg == 1 && sc.zero_bytes <= BK_SELF_CLEAR;
    if (!self) cudaMemsetAsync(sc.zero, 0, sc.zero_bytes, st);
    const int* route = nullptr;
    if (bk.on()) {
        bucket_launch<T>(d, tmp, want, p, bk, key_mask, out_mask, sc, self ? (uint32_t)(sc.zero_bytes / 16) : 0u, st);
        route = sc.route;
    }
    const Behind rest = behind(p, bk);
    if (rest == Behind::LEVELS) {
        const SegBucketPlan<T> q = behind_plan(p, bk);
        const SegBucketScratch<T> seg(scratch, q, reinterpret_cast<SbCounts*>(sc.err), false);
        const SbBuffers<T> buf{d, tmp, route, want == tmp};
        SbStarts plain{};
        if (bk.on() && sizeof(typename Traits<T>::Key) == 8)
            plain = SbStarts{bk.b2 ? sc.start2 : sc.start1, (uint32_t)bk.nbuckets, !bk.b2};
        const SbGiven given{route, sc.start1, p.n, p.len, (uint32_t)p.nseg, bk.b2 ? (uint32_t)(p.nseg << bk.b1) : 0u};
        segbucket_behind(buf, given, plain, q, key_mask, out_mask, seg, st);
        return cudaGetLastError();
    }
    if constexpr (sizeof(typename Traits<T>::Key) == 4) {
        if (rest == Behind::MERGES) {
            return sort_behind_u32(d, want, want == d ? tmp : d, want, n, sort_n, key_mask, out_mask, MERGES_CODE,
                                   scratch, route, sc.err, st);
        }
        if (p.wide)
            radix_launch<T, uint64_t>(d, tmp, want, p, sc, route, st);
        else
            radix_launch<T, uint32_t>(d, tmp, want, p, sc, route, st);
    }
    return cudaGetLastError();
}

}  // namespace origami
