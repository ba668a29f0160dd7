// Host launcher of the segmented bucket sort (seg_buckets.cuh).
#pragma once
#include <algorithm>
#include <string>

#include "pipeline.cuh"
#include "profiler.h"
#include "seg_buckets.cuh"

namespace origami {

// Geometry of the bucket sort of n items in segments whose lengths are on the device:
// none longer than `longest`, at most nseg shorter than a bucket.
template <class T>
struct SegBucketPlan {
    using Sh = SegBucketShape<T>;
    uint64_t n, nseg, segs, tiles, recs;
    int levels, usual;  // usual: what segments of the mean length need
    bool wide;  // 64-bit counts
    SegBucketPlan(uint64_t n_, uint64_t nseg_, uint64_t longest) : n(n_), nseg(nseg_) {
        // levels that splitters need to cut the longest segment into buckets of half the
        // largest size; from two levels on for four times fewer items, so that a key of some 9 % of
        // them does not send the first level to splitters (6,000,000 Zipf uint64 keys in two
        // levels, by splitters, 375 us, in three 233)
        levels = longest > (uint64_t)Sh::CAP ? 1 : 0;
        for (uint64_t m = (uint64_t)Sh::CAP / 2 << SB_SURE_BITS; levels && m < longest && levels < SB_MAX_LEVELS;
             m <<= levels == 2 ? SB_SURE_BITS - 2 : SB_SURE_BITS)
            ++levels;
        // many segments: their work, not the launches, decides, and slices of equal width are
        // the cheaper ones, so a level more than those need (2^26 normally distributed uint64
        // keys in segments of 2^17: one level by splitters 1.43 ms, two levels 0.95)
        if (levels && longest < n) {
            int wide = 2;
            for (uint64_t m = (uint64_t)Sh::CAP * 4 / 5 * RADIX_BINS; m < longest && wide < SB_MAX_LEVELS; m *= RADIX_BINS) ++wide;
            levels = std::max(levels, wide);
        }
        usual = 0;
        for (uint64_t m = (uint64_t)Sh::CAP * 4 / 5; m < n / std::max<uint64_t>(nseg, 1); m *= RADIX_BINS) ++usual;
        usual = std::max(usual, 1);
        // a level's segments are longer than a bucket
        segs = n / (Sh::CAP + 1) + 1;
        tiles = n / Sh::TILE + segs;
        // buckets, c = n / CAP: short segments; slices over half a bucket (2c); groups of
        // shorter ones (stretches of at least CAP / 3: 3c, one more in every segment of a
        // level: c a level, one more where a longer slice interrupts a stretch: 2c for
        // buckets, 2c a level for the next level's segments); pieces of equal keys (2c)
        recs = nseg + (10ull + 3 * (uint64_t)levels) * segs;
        // pairs keep two state bits beside their counts
        wide = n >= (Sh::STABLE ? 1ull << 30 : 1ull << 32);
    }
    bool fits() const { return tiles < (1ull << 31) && recs < (1ull << 31) && nseg < (1ull << 31); }
};

// Device scratch of one sort (each part 256-byte aligned); only the tail (the
// error word and the counters, SbCounts) has to start at 0.
template <class T>
struct SegBucketScratch {
    using K = typename Traits<T>::Key;
    uint64_t bytes = 0;
    SbSeg* list[2] = {nullptr, nullptr};
    SbMap<K>* maps = nullptr;
    K* splitters = nullptr;
    void* hist = nullptr;  // counts, then slice starts, then (keys) cursors
    uint32_t* done = nullptr;
    SbTile* tiles = nullptr;
    SbRec* recs = nullptr;
    uint32_t* slow = nullptr;
    void* look = nullptr;  // pairs
    SbCounts* cn = nullptr;
    // tail: where it is, if not here
    SegBucketScratch(void* base, const SegBucketPlan<T>& p, SbCounts* tail = nullptr, bool tail_here = true) {
        const uint64_t w = p.wide ? 8 : 4;
        char* b = static_cast<char*>(base);
        uint64_t o = 0;
        auto take = [&](uint64_t sz) {
            char* r = b ? b + o : nullptr;
            o += (sz + 255) & ~255ull;
            return r;
        };
        for (SbSeg*& l : list) l = reinterpret_cast<SbSeg*>(take(p.segs * sizeof(SbSeg)));
        maps = reinterpret_cast<SbMap<K>*>(take(p.segs * sizeof(SbMap<K>)));
        splitters = reinterpret_cast<K*>(take(p.segs * (SB_SPLITTERS + 1) * sizeof(K)));
        hist = take(p.segs * RADIX_BINS * w);
        done = reinterpret_cast<uint32_t*>(take(p.segs * 4));
        tiles = reinterpret_cast<SbTile*>(take(p.tiles * sizeof(SbTile)));
        recs = reinterpret_cast<SbRec*>(take(p.recs * sizeof(SbRec)));
        slow = reinterpret_cast<uint32_t*>(take(p.recs * 4));
        if (SegBucketShape<T>::STABLE) look = take(p.tiles * RADIX_BINS * w);
        cn = tail_here ? reinterpret_cast<SbCounts*>(take(256)) : tail;
        bytes = o;
    }
};

// Grids of the kernels, found once per process.
template <class T, class S>
struct SegBucketGrids {
    uint32_t sample, hist, pass, sort, rest;  // (rest: 32-bit keys)
    static const SegBucketGrids& get() {
        using Sh = SegBucketShape<T>;
        static const SegBucketGrids g = [] {
            SegBucketGrids r;
            r.sample = resident_ctas((const void*)sb_sample_kernel<T, S>, 512, 0);
            r.hist = resident_ctas((const void*)sb_hist_kernel<T, S>, 512, Sh::HIST_SMEM);
            if constexpr (Sh::STABLE)
                r.pass = resident_ctas((const void*)sb_stable_pass_kernel<T, S>, Sh::C::NT, Sh::PASS_SMEM);
            else {
                r.pass = resident_ctas((const void*)sb_pass_kernel<T, S, true>, Sh::C::NT, Sh::PASS_SMEM);
                resident_ctas((const void*)sb_pass_kernel<T, S, false>, Sh::C::NT, Sh::PASS_SMEM);
            }
            r.sort = resident_ctas((const void*)sb_sort_kernel<T, false>, Sh::Sort::C::S_NT, Sh::Sort::SORT_SMEM);
            if constexpr (sizeof(typename Traits<T>::Key) == 4)
                r.rest = resident_ctas((const void*)sb_sort_kernel<T, true>, Sh::Sort::C::S_NT, Sh::Sort::SORT_SMEM);
            return r;
        }();
        return g;
    }
};

// The levels and the bucket pass. given.nseg: behind a bucket sort that rarely gives up,
// where no level's grid is larger than resident; else for the segments in the first list,
// one CTA per tile on the levels that segments of the mean length need, a resident grid
// on those that few may (415M uint32 keys in 4096 segments: 0.33 ms of CTAs that found
// nothing to do).
template <class T, class S>
void segbucket_levels(const SbBuffers<T>& buf, const SbGiven& given, const SbStarts& plain, const SegBucketPlan<T>& p,
                      uint64_t xin, uint64_t xout, const SegBucketScratch<T>& sc, cudaStream_t st) {
    using Sh = SegBucketShape<T>;
    using K = typename Traits<T>::Key;
    using C = typename Sh::C;
    const SegBucketGrids<T, S>& g = SegBucketGrids<T, S>::get();
    static const std::string n_sample = std::string("segbucket_sample<") + TypeName<T>::v + ">";
    static const std::string n_hist = std::string("segbucket_hist<") + TypeName<T>::v + ">";
    static const std::string n_pass = std::string("segbucket_pass<") + TypeName<T>::v + ">";
    static const std::string n_sort = std::string("segbucket_sort<") + TypeName<T>::v + ">";
    SbCounts* cn = sc.cn;
    S* hist = static_cast<S*>(sc.hist);
    const bool behind = given.nseg != 0;
    const uint32_t segs = (uint32_t)p.segs, tiles = (uint32_t)p.tiles;
    for (int l = 0; l < p.levels; ++l) {
        SbHandOn to{};
        to.next = l + 1 < p.levels ? sc.list[(l + 1) & 1] : nullptr;
        to.next_count = &cn->segs[l + 1];
        to.recs = sc.recs;
        to.rec_count = &cn->recs;
        to.slow = sc.slow;
        to.stay = xin == xout;
        to.slow_count = &cn->slow;
        const SbGiven none{};
        const uint32_t samples = l == 0 && behind ? std::max(given.nseg, given.slices) : segs;
        launch(n_sample.c_str(), st, [&] {
            launch_dependent(sb_sample_kernel<T, S>, dim3(std::min(samples, g.sample)), dim3(512), 0, st, buf, l,
                             p.levels - 1 - l, l == 0 ? given : none, (const SbSeg*)sc.list[l & 1], &cn->segs[l], xin, sc.maps,
                             sc.splitters, hist, sc.done, sc.tiles, &cn->tiles[l], sc.recs, &cn->recs,
                             (const int*)&cn->err);
        });
        launch(n_hist.c_str(), st, [&] {
            launch_dependent(sb_hist_kernel<T, S>, dim3(std::min(tiles, g.hist)), dim3(512), Sh::HIST_SMEM, st, buf, l,
                             (const SbTile*)sc.tiles, (const uint32_t*)&cn->tiles[l], (const SbMap<K>*)sc.maps,
                             (const K*)sc.splitters, xin, hist, sc.done, to, static_cast<S*>(sc.look), &cn->err,
                             wait_limit());
        });
        launch(n_pass.c_str(), st, [&] {
            if constexpr (Sh::STABLE) {
                launch_dependent(sb_stable_pass_kernel<T, S>, dim3(std::min(tiles, g.pass)), dim3(C::NT), Sh::PASS_SMEM, st,
                                 buf, l, (const SbTile*)sc.tiles, (const uint32_t*)&cn->tiles[l],
                                 (const SbMap<K>*)sc.maps, (const K*)sc.splitters, xin, (const S*)hist,
                                 static_cast<S*>(sc.look), &cn->claim[l], &cn->err, wait_limit());
            } else {
                const bool loop = behind || l >= p.usual;
                launch_dependent(loop ? sb_pass_kernel<T, S, true> : sb_pass_kernel<T, S, false>,
                                 dim3(loop ? std::min(tiles, g.pass) : tiles), dim3(C::NT), Sh::PASS_SMEM, st, buf, l,
                                 (const SbTile*)sc.tiles, (const uint32_t*)&cn->tiles[l], (const SbMap<K>*)sc.maps,
                                 (const K*)sc.splitters, xin, hist, (const int*)&cn->err);
            }
        });
    }
    auto sort = [&](auto kernel, uint32_t grid, uint32_t first) {
        launch(n_sort.c_str(), st, [&] {
            launch_dependent(kernel, dim3(grid), dim3(Sh::Sort::C::S_NT), Sh::Sort::SORT_SMEM, st, buf, plain,
                             (const SbRec*)sc.recs, (const uint32_t*)sc.slow, (const SbCounts*)cn, first, xin, xout);
        });
    };
    if constexpr (sizeof(K) == 4)
        if (behind) return sort(sb_sort_kernel<T, true>, g.rest, 0u);
    // one CTA per bucket: neighbouring buckets of a segment hold more than CAP items
    // together, so few sorts have more than these, and few CTAs stand by for the rest
    const uint32_t first = (uint32_t)std::min(p.recs, std::max<uint64_t>(plain.buckets, p.nseg + p.n * 9 / (4 * (uint64_t)Sh::CAP) + 1));
    sort(sb_sort_kernel<T, false>, std::max(first, plain.buckets) + std::min(first, g.sort / 4), first);
}

// The levels as what stands behind a bucket sort (radix_host.cuh). Defined with the
// segmented sort, in seg_bucket_*.cu: a kernel is launched from one translation unit only,
// since each has a copy of it, and what is set once per process (shared-memory limits,
// grids) is set for one copy.
#define ORIGAMI_DECLARE_BEHIND(T)                                                                                        \
    void segbucket_behind(const SbBuffers<T>& buf, const SbGiven& given, const SbStarts& plain, const SegBucketPlan<T>& p, \
                          uint64_t xin, uint64_t xout, const SegBucketScratch<T>& sc, cudaStream_t st);
ORIGAMI_DECLARE_BEHIND(uint32_t)
ORIGAMI_DECLARE_BEHIND(uint64_t)
ORIGAMI_DECLARE_BEHIND(KV64)
#undef ORIGAMI_DECLARE_BEHIND

template <class T>
void segbucket_run(const SbBuffers<T>& buf, const SbGiven& given, const SbStarts& plain, const SegBucketPlan<T>& p,
                   uint64_t xin, uint64_t xout, const SegBucketScratch<T>& sc, cudaStream_t st) {
    if (p.wide)
        segbucket_levels<T, uint64_t>(buf, given, plain, p, xin, xout, sc, st);
    else
        segbucket_levels<T, uint32_t>(buf, given, plain, p, xin, xout, sc, st);
}

// Segments [off[s], off[s+1]), sorted in place.
template <class T>
cudaError_t segbucket_run(T* d, T* tmp, const uint64_t* off, uint64_t nseg, uint64_t n, uint64_t xmask, void* scratch,
                          cudaStream_t st) {
    const SegBucketPlan<T> p(n, nseg, n);
    const SegBucketScratch<T> sc(scratch, p);
    static const std::string n_plan = std::string("segbucket_plan<") + TypeName<T>::v + ">";
    cudaMemsetAsync(sc.cn, 0, 256, st);
    launch(n_plan.c_str(), st, [&] {
        sb_plan_kernel<T><<<(unsigned)((nseg + 255) / 256), 256, 0, st>>>(off, (uint32_t)nseg, n, sc.list[0],
                                                                         (uint32_t)p.segs, sc.recs, sc.cn);
    });
    segbucket_run<T>(SbBuffers<T>{d, tmp, nullptr, false}, SbGiven{}, SbStarts{}, p, xmask, xmask, sc, st);
    return cudaGetLastError();
}

}  // namespace origami
