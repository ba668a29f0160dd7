// Host launcher of the segmented bucket sort (seg_buckets.cuh).
#pragma once
#include <algorithm>
#include <string>

#include "pipeline.cuh"
#include "profiler.h"
#include "radix_host.cuh"
#include "seg_buckets.cuh"

namespace origami {

// Geometry of the bucket sort of nseg segments of n items in all; their lengths
// are on the device.
template <class T>
struct SegBucketPlan {
    using Sh = SegBucketShape<T>;
    uint64_t n, nseg, segs, tiles, recs;
    int levels;
    bool wide;  // 64-bit counts
    SegBucketPlan(uint64_t n_, uint64_t nseg_) : n(n_), nseg(nseg_) {
        // levels that 256 slices each need to cut one segment of n items into buckets
        // of 4/5 of the largest size, and one more for keys that are spread unevenly
        levels = 1;
        for (uint64_t m = (uint64_t)Sh::CAP * 4 / 5 * RADIX_BINS; m < n && levels < SB_MAX_LEVELS; m *= RADIX_BINS) ++levels;
        levels = n > (uint64_t)Sh::CAP ? std::min(levels + 1, SB_MAX_LEVELS) : 0;
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
    uint64_t bytes = 0, tail_at = 0;
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
    SegBucketScratch(void* base, const SegBucketPlan<T>& p) {
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
        tail_at = o;
        cn = reinterpret_cast<SbCounts*>(take(256));
        bytes = o;
    }
};

// Grids of the kernels, found once per process.
template <class T, class S>
struct SegBucketGrids {
    uint32_t sample, hist, pass, rest;
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
            resident_ctas((const void*)sb_sort_kernel<T>, Sh::Sort::C::S_NT, Sh::Sort::SORT_SMEM);
            r.rest = resident_ctas((const void*)sb_rest_kernel<T>, Sh::Sort::C::S_NT, Sh::Sort::SORT_SMEM);
            return r;
        }();
        return g;
    }
};

template <class T, class S>
cudaError_t segbucket_launch(T* d, T* tmp, const SegBucketPlan<T>& p, const uint64_t* off, uint64_t xmask,
                             const SegBucketScratch<T>& sc, cudaStream_t st) {
    using Sh = SegBucketShape<T>;
    using K = typename Traits<T>::Key;
    using C = typename Sh::C;
    const SegBucketGrids<T, S>& g = SegBucketGrids<T, S>::get();
    static const std::string n_plan = std::string("segbucket_plan<") + TypeName<T>::v + ">";
    static const std::string n_sample = std::string("segbucket_sample<") + TypeName<T>::v + ">";
    static const std::string n_hist = std::string("segbucket_hist<") + TypeName<T>::v + ">";
    static const std::string n_pass = std::string("segbucket_pass<") + TypeName<T>::v + ">";
    static const std::string n_sort = std::string("segbucket_sort<") + TypeName<T>::v + ">";
    static const std::string n_rest = std::string("segbucket_rest<") + TypeName<T>::v + ">";
    SbCounts* cn = sc.cn;
    S* hist = static_cast<S*>(sc.hist);
    const uint32_t segs = (uint32_t)p.segs, tiles = (uint32_t)p.tiles;
    cudaMemsetAsync(cn, 0, 256, st);
    launch(n_plan.c_str(), st, [&] {
        sb_plan_kernel<T><<<(unsigned)((p.nseg + 255) / 256), 256, 0, st>>>(off, (uint32_t)p.nseg, p.n, sc.list[0], segs,
                                                                           sc.recs, cn);
    });
    for (int l = 0; l < p.levels; ++l) {
        const T* src = (l & 1) ? tmp : d;
        T* dst = (l & 1) ? d : tmp;
        SbHandOn to;
        to.next = l + 1 < p.levels ? sc.list[(l + 1) & 1] : nullptr;
        to.next_count = &cn->segs[l + 1];
        to.recs = sc.recs;
        to.rec_count = &cn->recs;
        to.flags = dst == tmp ? SbRec::TMP : 0;
        to.stay = dst == d;
        launch(n_sample.c_str(), st, [&] {
            launch_dependent(sb_sample_kernel<T, S>, dim3(std::min(segs, g.sample)), dim3(512), 0, st, src,
                             (const SbSeg*)sc.list[l & 1], (const uint32_t*)&cn->segs[l], xmask, sc.maps, sc.splitters,
                             hist, sc.done, sc.tiles, &cn->tiles[l], (const int*)&cn->err);
        });
        launch(n_hist.c_str(), st, [&] {
            launch_dependent(sb_hist_kernel<T, S>, dim3(std::min(tiles, g.hist)), dim3(512), Sh::HIST_SMEM, st, src,
                             (const SbTile*)sc.tiles, (const uint32_t*)&cn->tiles[l], (const SbMap<K>*)sc.maps,
                             (const K*)sc.splitters, xmask, hist, sc.done, to, static_cast<S*>(sc.look), &cn->err,
                             wait_limit());
        });
        launch(n_pass.c_str(), st, [&] {
            if constexpr (Sh::STABLE) {
                launch_dependent(sb_stable_pass_kernel<T, S>, dim3(std::min(tiles, g.pass)), dim3(C::NT), Sh::PASS_SMEM, st,
                                 src, dst, (const SbTile*)sc.tiles, (const uint32_t*)&cn->tiles[l],
                                 (const SbMap<K>*)sc.maps, (const K*)sc.splitters, xmask, (const S*)hist,
                                 static_cast<S*>(sc.look), &cn->claim[l], &cn->err, wait_limit());
            } else {
                const bool loop = l > 0 && l + 1 == p.levels;
                launch_dependent(loop ? sb_pass_kernel<T, S, true> : sb_pass_kernel<T, S, false>,
                                 dim3(loop ? std::min(tiles, g.pass) : tiles), dim3(C::NT), Sh::PASS_SMEM, st, src, dst,
                                 (const SbTile*)sc.tiles, (const uint32_t*)&cn->tiles[l], (const SbMap<K>*)sc.maps,
                                 (const K*)sc.splitters, xmask, hist, (const int*)&cn->err);
            }
        });
    }
    // one CTA per bucket. Neighbouring buckets of a segment hold more than CAP items
    // together, so few sorts have more than these; sb_rest_kernel takes the others
    const uint32_t first = (uint32_t)std::min(p.recs, p.nseg + p.n * 9 / (4 * (uint64_t)Sh::CAP) + 1);
    launch(n_sort.c_str(), st, [&] {
        launch_dependent(sb_sort_kernel<T>, dim3(first), dim3(Sh::Sort::C::S_NT), Sh::Sort::SORT_SMEM, st, d, tmp,
                         (const SbRec*)sc.recs, sc.slow, cn, xmask);
    });
    launch(n_rest.c_str(), st, [&] {
        launch_dependent(sb_rest_kernel<T>, dim3((unsigned)std::min<uint64_t>(p.recs, g.rest)), dim3(Sh::Sort::C::S_NT),
                         Sh::Sort::SORT_SMEM, st, d, tmp, (const SbRec*)sc.recs, (const uint32_t*)sc.slow, (const SbCounts*)cn,
                         first, xmask);
    });
    return cudaGetLastError();
}

template <class T>
cudaError_t segbucket_run(T* d, T* tmp, const uint64_t* off, uint64_t nseg, uint64_t n, uint64_t xmask, void* scratch,
                          cudaStream_t st) {
    const SegBucketPlan<T> p(n, nseg);
    const SegBucketScratch<T> sc(scratch, p);
    if (p.wide) return segbucket_launch<T, uint64_t>(d, tmp, p, off, xmask, sc, st);
    return segbucket_launch<T, uint32_t>(d, tmp, p, off, xmask, sc, st);
}

}  // namespace origami
