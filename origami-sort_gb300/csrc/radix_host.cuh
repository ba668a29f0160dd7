// Host launcher of the radix passes (radix.cuh).
#pragma once
#include <algorithm>
#include <string>

#include "pipeline.cuh"
#include "profiler.h"
#include "radix.cuh"

namespace origami {

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
    // Whole tiles per segment, and tile numbers that fit 31 bits.
    static bool fits(uint64_t n, uint64_t sort_n) {
        const uint64_t len = chunk_limit(n, sort_n);
        return n >= 2 && (len == n || len % Sh::TILE == 0) && n / Sh::TILE < (1ull << 31) - 2;
    }
};

// Device scratch of one radix sort (each part 256-byte aligned):
//   look 0/1   look-back words of the even / odd passes, 256 per tile
//   hist       digit counts, [segment][digit][256]
//   tail       256 bytes: the error word, the passes' tile counters (+64)
// hist and tail start at zero (one memset).
template <class T>
struct RadixScratch {
    uint64_t bytes = 0, zero_bytes = 0;
    void* look[2] = {nullptr, nullptr};
    void* hist = nullptr;
    int* err = nullptr;
    unsigned* claim = nullptr;
    RadixScratch(void* base, const RadixPlan<T>& p) {
        const uint64_t w = p.wide ? 8 : 4;
        char* b = static_cast<char*>(base);
        uint64_t o = 0;
        auto take = [&](uint64_t sz) {
            char* r = b ? b + o : nullptr;
            o += (sz + 255) & ~255ull;
            return r;
        };
        for (void*& l : look) l = take(p.tiles * RADIX_BINS * w);
        zero_bytes = o;
        hist = take(p.nseg * RadixShape<T>::DIGITS * RADIX_BINS * w);
        err = reinterpret_cast<int*>(take(256));
        claim = b ? reinterpret_cast<unsigned*>(reinterpret_cast<char*>(err) + 64) : nullptr;
        zero_bytes = o - zero_bytes;
        bytes = o;
    }
};

template <class T>
uint64_t radix_scratch_bytes(uint64_t n, uint64_t sort_n) {
    return RadixScratch<T>(nullptr, RadixPlan<T>(n, sort_n)).bytes;
}

template <class T, class S>
cudaError_t radix_launch(T* d, T* other, bool copy, const RadixPlan<T>& p, uint64_t xmask, const RadixScratch<T>& sc,
                         cudaStream_t st) {
    using Sh = RadixShape<T>;
    using G = RadixUniform;
    struct Grids {
        uint32_t hist, pass;
    };
    static const Grids g = [] {  // kernel attributes and grids, once per process
        int dev = 0, sms = 0, per = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaFuncSetAttribute(radix_pass_kernel<T, S, G>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Sh::SMEM);
        cudaFuncSetAttribute(radix_hist_kernel<T, S, G, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)Sh::HIST_SMEM);
        cudaFuncSetAttribute(radix_hist_kernel<T, S, G, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)Sh::HIST_SMEM);
        Grids r;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, radix_hist_kernel<T, S, G, false>, 512, Sh::HIST_SMEM);
        r.hist = (uint32_t)(sms * (per > 0 ? per : 1));
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, radix_pass_kernel<T, S, G>, Sh::NT, Sh::SMEM);
        r.pass = (uint32_t)(sms * (per > 0 ? per : 1));
        return r;
    }();
    static const std::string n_hist = std::string("radix_hist<") + TypeName<T>::v + ">";
    static const std::string n_pass = std::string("radix_pass<") + TypeName<T>::v + ">";
    const uint32_t tiles = (uint32_t)p.tiles;
    const G geo{p.n, p.len, p.shift};
    S* hist = static_cast<S*>(sc.hist);
    cudaMemsetAsync(hist, 0, sc.zero_bytes, st);
    launch(n_hist.c_str(), st, [&] {
        const uint32_t gh = std::min(tiles, g.hist);
        S* l0 = static_cast<S*>(sc.look[0]);
        if (copy)
            radix_hist_kernel<T, S, G, true><<<gh, 512, Sh::HIST_SMEM, st>>>(d, other, geo, tiles, xmask, hist, l0);
        else
            radix_hist_kernel<T, S, G, false><<<gh, 512, Sh::HIST_SMEM, st>>>(d, nullptr, geo, tiles, xmask, hist, l0);
    });
    T* src = copy ? other : d;
    T* dst = copy ? d : other;
    static_assert(Sh::DIGITS % 2 == 0, "the passes end in the buffer they start from");
    for (int b = 0; b < Sh::DIGITS; ++b) {
        launch(n_pass.c_str(), st, [&] {
            launch_dependent(radix_pass_kernel<T, S, G>, dim3(std::min(tiles, g.pass)), dim3(Sh::NT), Sh::SMEM, st,
                             (const T*)src, dst, geo, tiles, b, xmask, (const S*)hist, static_cast<S*>(sc.look[b & 1]),
                             b + 1 < Sh::DIGITS ? static_cast<S*>(sc.look[(b + 1) & 1]) : (S*)nullptr, sc.claim + b,
                             sc.err, wait_limit());
        });
        std::swap(src, dst);
    }
    return cudaGetLastError();
}

// Sorts d[0..n) in chunks of sort_n (0 = one full sort) into `want` (d or tmp).
// The passes are an even number, so they end in the buffer they start from:
// with want == tmp the counting kernel copies the input there as it reads it.
// `scratch` holds radix_scratch_bytes<T>(n, sort_n) bytes.
template <class T>
cudaError_t radix_sort(T* d, T* tmp, uint64_t n, uint64_t sort_n, uint64_t key_mask, T* want, void* scratch,
                       cudaStream_t st) {
    const RadixPlan<T> p(n, sort_n);
    const RadixScratch<T> sc(scratch, p);
    if (p.wide) return radix_launch<T, uint64_t>(d, tmp, want == tmp, p, key_mask, sc, st);
    return radix_launch<T, uint32_t>(d, tmp, want == tmp, p, key_mask, sc, st);
}

}  // namespace origami
