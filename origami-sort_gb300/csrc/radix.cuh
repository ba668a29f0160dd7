// Radix passes: what device sorts of 32-bit keys with min_k = 0 use where the bucket
// sort (buckets.cuh) does not take the call or gives up; its partition of pairs is
// the pass kernel here.
//
// A merge level moves every item once through HBM and doubles the runs; a
// radix pass moves every item once and settles eight bits of the key, whatever
// the length. 2^28 uint32 keys take 4 passes and one read for the digit counts
// instead of 16 merge passes. The passes go from the lowest digit to the
// highest and each is stable, so the result is the stable sort: byte for byte
// what the merge pipeline produces.
//
//   radix_hist_kernel  one read of the input counts every digit of every key,
//                      per segment (a segment is the whole array or one chunk)
//   radix_pass_kernel  one pass over one digit, single read and single write
//                      (the "onesweep" scheme, Adinets and Merrill 2022, with
//                      the decoupled look-back of Merrill and Garland 2016)
//
// A pass works on tiles of NT * IPT items. A CTA claims a tile, holds its items
// in registers, counts their digits (every 16 lanes against 256 words of their
// own), publishes the tile's counts, places the items in digit order in shared
// memory, and learns where each digit's items go by looking back over the
// counts of the tiles before it until it meets one that already knows its
// prefix. The first tile of a segment starts from the scanned digit counts.
// Tiles are claimed in order, so the tiles a look-back waits for are always
// held by running CTAs.
//
// Ranking. A word holds the next place of a digit (upper half) and, during a
// step, which of the 16 lanes have it (lower half): one shared-memory OR, one
// load, a population count, one store by the digit's last lane: 8 cycles per
// warp step and SM. Ballots over the eight bits take 13 to 26, match.any 61. A
// digit that holds more than 1/24 of the segment would serialise the atomics
// (32 equal lanes: 36 cycles), so such passes take the ballots; a digit that
// holds the whole segment makes the pass a plain copy.
//
// What bounds it (2^28 uint32 keys, one GB300): the shared-memory pipe. A step
// of 32 keys costs about 25 cycles of it (five random accesses of 3.5 bank
// conflicts each), 0.86 ms a pass against 0.32 ms of HBM traffic. Whole sorts:
// 1 GiB uint32 7.38 ms by merges, 3.79 by radix passes alone.
//
// Every wait is bounded (`spin` polls): on expiry the CTA records
// ERR_WAIT_EXPIRED and stops, waiting CTAs see the word and stop, later passes
// return at once. No bulk copies are involved, so nothing is left in flight.
#pragma once
#include <cstdint>

#include "bulk.cuh"
#include "common.cuh"

namespace origami {

constexpr int RADIX_BITS = 8;
constexpr int RADIX_BINS = 1 << RADIX_BITS;

template <class T>
struct RadixCfg;
template <>
struct RadixCfg<uint32_t> {
    static constexpr int NT = 256, IPT = 32, MINB = 3;  // tile: 8192 keys, 32 KiB
    static constexpr int HIST_COPIES = 8;
};
template <>
struct RadixCfg<uint64_t> {  // (whole tiles a chunk only)
    static constexpr int NT = 256, IPT = 16, MINB = 3;  // 4096 keys, 32 KiB
};
template <>
struct RadixCfg<KV64> {  // (the partition of the bucket sort)
    static constexpr int NT = 256, IPT = 16, MINB = 2;  // 4096 pairs, 64 KiB
};

template <class T>
struct RadixShape {
    using C = RadixCfg<T>;
    static constexpr int NT = C::NT, IPT = C::IPT, NG = NT / 16;
    static constexpr int TILE = NT * IPT;
    static constexpr int DIGITS = (int)sizeof(typename Traits<T>::Key);  // 8-bit digits of a key
    static constexpr size_t KEYS_BYTES = (size_t)TILE * sizeof(T);
    static constexpr size_t SMEM = KEYS_BYTES + (size_t)NG * RADIX_BINS * 4;
    static_assert(NT >= RADIX_BINS, "one thread per bin");
};

// Digit `byte` of a key.
__device__ __forceinline__ unsigned radix_digit(uint32_t k, int byte) { return __byte_perm(k, 0, 0x4440 | byte); }

// Lanes of the warp whose digit equals this lane's: eight ballots, each turned
// round where this lane's bit is 0. (Written as PTX: from C++ the same ballots
// took 24 cycles per step and SM instead of 12; match.any took 60.)
__device__ __forceinline__ unsigned radix_match(unsigned d) {
    unsigned m = 0xFFFFFFFFu;
#pragma unroll
    for (int b = 0; b < RADIX_BITS; ++b) {
        unsigned r;
        asm volatile(
            "{\n .reg .pred p;\n .reg .b32 t, x;\n and.b32 t, %1, %2;\n setp.ne.u32 p, t, 0;\n"
            " vote.sync.ballot.b32 x, p, 0xffffffff;\n @!p not.b32 x, x;\n mov.b32 %0, x;\n}\n"
            : "=r"(r)
            : "r"(d), "r"(1u << b));
        m &= r;
    }
    return m;
}

// Look-back words: a count with a state in its two top bits. 32-bit words serve
// segments of fewer than 2^30 items, 64-bit words longer ones.
template <class S>
struct LookWord {
    static constexpr int SH = (int)sizeof(S) * 8 - 2;
    static constexpr S MASK = (S(1) << SH) - 1;
    static constexpr S COUNT = S(1) << SH;   // the tile's own count
    static constexpr S PREFIX = S(2) << SH;  // count of everything before and in the tile
};
__device__ __forceinline__ uint32_t look_load(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint64_t look_load(const uint64_t* p) {
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];\n" : "=l"(v) : "l"(p) : "memory");
    return v;
}
// The route word of a bucket sort (buckets.cuh): from L2, because kernels that
// overlap (programmatic dependent launch) read it while one of them may set it.
__device__ __forceinline__ int route_load(const int* p) {
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void look_store(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;\n" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void look_store(uint64_t* p, uint64_t v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;\n" ::"l"(p), "l"(v) : "memory");
}

// Segments of equal length `len` (a power of two and a multiple of the tile, or
// the whole array as one segment): tile t belongs to segment t >> shift.
struct RadixUniform {
    uint64_t n, len;
    uint32_t shift;  // log2(tiles per segment); 31: one segment
    struct Tile {
        uint64_t base, sbase, slen;  // first item; the segment's first item and length
        uint32_t seg, ti;            // segment; the tile's number inside it
        int cnt;                     // items in the tile
    };
    __device__ __forceinline__ uint32_t total(uint32_t tiles) const { return tiles; }
    template <int TILE>
    __device__ __forceinline__ Tile tile(uint32_t t) const {
        Tile r;
        r.seg = t >> shift;
        r.ti = t - (r.seg << shift);
        r.sbase = (uint64_t)r.seg * len;
        r.base = (uint64_t)t * TILE;
        r.slen = n - r.sbase < len ? n - r.sbase : len;
        const uint64_t rest = r.slen - (uint64_t)r.ti * TILE;
        r.cnt = (int)(rest < (uint64_t)TILE ? rest : (uint64_t)TILE);
        return r;
    }
};

// Counts every digit of every key: hist[segment][digit][bin] += count. Each
// warp's lanes spread over HIST_COPIES copies of the counters, so that lanes
// with equal digits mostly meet different banks. A CTA takes a contiguous range
// of tiles and flushes its counters when the segment changes. Also clears the
// first pass's look-back words, and copies the input to `want` where it is not
// there yet (the passes are an even number and end where they start).
// route (optional): the radix passes stand behind a bucket sort (buckets.cuh);
// 0: it has done the work, return; 2: the items are in `moved` instead of `in`.
template <class T>
constexpr size_t radix_hist_smem() {
    return (size_t)RadixShape<T>::DIGITS * RADIX_BINS * RadixCfg<T>::HIST_COPIES * 4;
}
template <class T, class S, class G>
__global__ void __launch_bounds__(512) radix_hist_kernel(const T* in0, const T* moved, T* want, G geo, uint32_t tiles,
                                                         S* hist, S* look0, const int* route) {
    using Sh = RadixShape<T>;
    constexpr int D = Sh::DIGITS, C = Sh::C::HIST_COPIES, TILE = Sh::TILE;
    extern __shared__ __align__(16) uint32_t cnt_sm[];
    const int tid = threadIdx.x, col = tid & (C - 1);
    grid_dep_wait();
    const int r = route ? route_load(route) : 1;
    if (r == 0) return;
    const T* in = r == 2 ? moved : in0;
    const bool copy = in != want;
    const uint32_t t0 = (uint32_t)((uint64_t)tiles * blockIdx.x / gridDim.x);
    const uint32_t t1 = (uint32_t)((uint64_t)tiles * (blockIdx.x + 1) / gridDim.x);
    for (int i = tid; i < D * RADIX_BINS * C; i += 512) cnt_sm[i] = 0;
    __syncthreads();
    auto flush = [&](uint32_t seg) {
        __syncthreads();
        for (int i = tid; i < D * RADIX_BINS; i += 512) {
            uint32_t s = 0;
#pragma unroll
            for (int c = 0; c < C; ++c) {
                s += cnt_sm[i * C + c];
                cnt_sm[i * C + c] = 0;
            }
            if (s) {
                if constexpr (sizeof(S) == 8)
                    atomicAdd(reinterpret_cast<unsigned long long*>(hist) + (size_t)seg * D * RADIX_BINS + i,
                              (unsigned long long)s);
                else
                    atomicAdd(hist + (size_t)seg * D * RADIX_BINS + i, s);
            }
        }
        __syncthreads();
    };
    auto count = [&](const T& v) {
        const auto k = Traits<T>::key(v);
#pragma unroll
        for (int b = 0; b < D; ++b) atomicAdd(&cnt_sm[(b * RADIX_BINS + radix_digit(k, b)) * C + col], 1u);
    };
    uint32_t seg = 0xFFFFFFFFu;
    for (uint32_t t = t0; t < t1; ++t) {
        const auto q = geo.template tile<TILE>(t);
        if (q.seg != seg) {
            if (seg != 0xFFFFFFFFu) flush(seg);
            seg = q.seg;
        }
        constexpr int V = Vec<T>::N;
        const T* p = in + q.base;
        const int nvec = q.cnt / V;  // tiles start 16-byte aligned
        if (q.cnt == TILE) {
#pragma unroll
            for (int j = 0; j < TILE / V / 512; ++j) {
                const int i = j * 512 + tid;
                const uint4 x = reinterpret_cast<const uint4*>(p)[i];
                if (copy) reinterpret_cast<uint4*>(want + q.base)[i] = x;
                const T* e = reinterpret_cast<const T*>(&x);
#pragma unroll
                for (int k = 0; k < V; ++k) count(e[k]);
            }
        } else {
            for (int i = tid; i < nvec; i += 512) {
                const uint4 x = reinterpret_cast<const uint4*>(p)[i];
                if (copy) reinterpret_cast<uint4*>(want + q.base)[i] = x;
                const T* e = reinterpret_cast<const T*>(&x);
#pragma unroll
                for (int k = 0; k < V; ++k) count(e[k]);
            }
            for (int i = nvec * V + tid; i < q.cnt; i += 512) {
                const T x = p[i];
                if (copy) want[q.base + i] = x;
                count(x);
            }
        }
        for (int i = tid; i < RADIX_BINS; i += 512) look0[(size_t)t * RADIX_BINS + i] = 0;
    }
    if (seg != 0xFFFFFFFFu) flush(seg);
}

// Exclusive scan over the 256 bins (one value per thread of the first 8 warps;
// `ws` is 8 values of scratch). Every thread of the CTA calls it. One barrier inside,
// and `ws` is read behind it: it is free again only after another one.
template <class S>
__device__ __forceinline__ S radix_bin_scan(S v, S* ws) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    S inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const S u = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= o) inc += u;
    }
    if (lane == 31 && warp < RADIX_BINS / 32) ws[warp] = inc;
    __syncthreads();
    S base = 0;
#pragma unroll
    for (int w = 0; w < RADIX_BINS / 32; ++w)
        if (w < warp) base += ws[w];
    return base + inc - v;
}

// The digit of a radix pass: byte `byte` of the key. Also what a pass asks about
// its segments: the count of a bin, and where the bin starts in the segment.
template <class T, class S>
struct ByteDigit {
    static constexpr bool kHeavy = true;  // any share of the items may have one digit
    const S* hist;
    int byte;
    ByteDigit(const S* h, int b) : hist(h), byte(b) {}
    __device__ __forceinline__ unsigned operator()(const T& v) const { return radix_digit(Traits<T>::key(v), byte); }
    __device__ __forceinline__ void enter(uint32_t) {}  // a tile of this segment follows
    __device__ __forceinline__ S count(uint32_t seg, int bin) const {
        return hist[((size_t)seg * RadixShape<T>::DIGITS + byte) * RADIX_BINS + bin];
    }
    // every thread of the CTA calls it (a barrier inside)
    __device__ __forceinline__ S first(uint32_t seg, uint64_t, S* ws) const {
        const int bin = threadIdx.x;
        return radix_bin_scan<S>(bin < RADIX_BINS ? count(seg, bin) : (S)0, ws);
    }
};

// One pass: src -> dst by one digit. look: this pass's words, 256 per tile, zero
// at launch; look_next (optional): the next pass's, cleared here. route
// (optional): run only where it holds `run` (radix passes behind a bucket sort
// run unless it is 0, the stable partition of a bucket sort while it is 0). (No early start of the next pass: its waiting
// CTAs cost more than its launch, 2^20 uint32 Zipf keys 0.078 ms without and 0.111 with.)
template <class T, class S, class G, class D>
__global__ void __launch_bounds__(RadixCfg<T>::NT, RadixCfg<T>::MINB)
    radix_pass_kernel(const T* src, T* dst, G geo, uint32_t tiles, D digit, S* look,
                      S* look_next, unsigned* claim, int* err, uint32_t spin,
                      const int* route, bool buckets) {
    using Sh = RadixShape<T>;
    using W = LookWord<S>;
    constexpr int NT = Sh::NT, IPT = Sh::IPT, NG = Sh::NG, TILE = Sh::TILE;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* skeys = reinterpret_cast<T*>(smem_raw);
    uint32_t* table = reinterpret_cast<uint32_t*>(smem_raw + Sh::KEYS_BYTES);  // [NG][256]
    __shared__ S goff[RADIX_BINS];
    __shared__ uint32_t ws[RADIX_BINS / 32];
    __shared__ S ws2[RADIX_BINS / 32];
    __shared__ uint32_t next_tile;
    const int tid = threadIdx.x, hl = tid & 15, grp = tid >> 4;
    uint32_t* gt = table + grp * RADIX_BINS;
    const unsigned one = 1u << hl, lt = one - 1u;

    grid_dep_wait();
    if (route && (route_load(route) == 0) != buckets) return;
    tiles = geo.total(tiles);
    if (tid == 0) next_tile = atomicAdd(claim, 1u);
    if (__syncthreads_or(tid == 0 && err_wait_set(err))) return;
    uint32_t t = next_tile, seg = 0xFFFFFFFFu;
    bool heavy = false;
    for (; t < tiles; t = next_tile) {
        const typename G::Tile q = geo.template tile<TILE>(t);
        if (q.seg != seg) digit.enter(q.seg);
        if (D::kHeavy && q.seg != seg) {
            const S h = tid < RADIX_BINS ? digit.count(q.seg, tid) : (S)0;
            heavy = __syncthreads_or(h > (S)(q.slen / 24));
            if (heavy && __syncthreads_or(h == (S)q.slen)) {
                // one digit only: the segment keeps its order. (A tile of it
                // takes no part in the look-back, like all the others.)
                for (int i = tid; i < q.cnt; i += NT) dst[q.base + i] = src[q.base + i];
                if (look_next)
                    for (int i = tid; i < RADIX_BINS; i += NT) look_next[(size_t)t * RADIX_BINS + i] = 0;
                if (tid == 0) next_tile = atomicAdd(claim, 1u);
                __syncthreads();
                continue;
            }
        }
        seg = q.seg;
        T v[IPT];
        const int i0 = grp * (16 * IPT) + hl;
        const int mine = q.cnt - i0;  // item i of this thread exists when i * 16 < mine
        {
            const T* p = src + q.base;
            if (q.cnt == TILE) {
#pragma unroll
                for (int i = 0; i < IPT; ++i) v[i] = p[i0 + i * 16];
            } else {
#pragma unroll
                for (int i = 0; i < IPT; ++i) v[i] = p[min(i0 + i * 16, q.cnt - 1)];
            }
        }
        {
            uint4* z = reinterpret_cast<uint4*>(gt);
#pragma unroll
            for (int i = 0; i < RADIX_BINS / 64; ++i) z[i * 16 + hl] = make_uint4(0, 0, 0, 0);
        }
        __syncwarp();
        // lanes of the group whose item of step i exists
        auto present = [&](int i) -> unsigned {
            const int k = min(max(mine + hl - i * 16, 0), 16);
            return 0xFFFFu >> (16 - k);
        };
        // count the group's digits (upper half of its words)
        if (!D::kHeavy || !heavy) {
#pragma unroll
            for (int i = 0; i < IPT; ++i)
                if (i * 16 < mine) atomicAdd(&gt[digit(v[i])], 1u << 16);
        } else {
#pragma unroll
            for (int i = 0; i < IPT; ++i) {
                const unsigned d = digit(v[i]);
                const unsigned m = (radix_match(d) >> (tid & 16)) & present(i);
                if ((m & one) && !(m & lt)) atomicAdd(&gt[d], (unsigned)__popc(m) << 16);
            }
        }
        __syncthreads();
        // per bin: the tile's count, published, and the groups' first places
        uint32_t total = 0;
        S* my = look + (size_t)t * RADIX_BINS + tid;
        if (tid < RADIX_BINS) {
#pragma unroll
            for (int g = 0; g < NG; ++g) total += table[g * RADIX_BINS + tid] >> 16;
            if (q.ti) look_store(my, W::COUNT | (S)total);
            if (look_next) look_next[(size_t)t * RADIX_BINS + tid] = 0;
        }
        const uint32_t start = radix_bin_scan<uint32_t>(total, ws);
        if (tid < RADIX_BINS) {
            uint32_t run = start;
#pragma unroll
            for (int g = 0; g < NG; ++g) {
                const uint32_t c = table[g * RADIX_BINS + tid] >> 16;
                table[g * RADIX_BINS + tid] = run << 16;
                run += c;
            }
        }
        __syncthreads();
        // rank and order the tile by digit in shared memory
        if (!D::kHeavy || !heavy) {
#pragma unroll
            for (int i = 0; i < IPT; ++i) {
                const unsigned d = digit(v[i]);
                if (i * 16 < mine) atomicOr(&gt[d], one);
                __syncwarp();
                const uint32_t w = gt[d], m = w & 0xFFFFu;
                const uint32_t r = (w >> 16) + __popc(m & lt);
                __syncwarp();
                if ((m >> hl) == 1u) gt[d] = (r + 1) << 16;  // the digit's last lane
                __syncwarp();
                if (i * 16 < mine) skeys[r] = v[i];
            }
        } else {
#pragma unroll
            for (int i = 0; i < IPT; ++i) {
                const unsigned d = digit(v[i]);
                const unsigned m = (radix_match(d) >> (tid & 16)) & present(i);
                const uint32_t r = (gt[d] >> 16) + __popc(m & lt);
                __syncwarp();
                if ((m >> hl) == 1u) gt[d] = (r + 1) << 16;
                __syncwarp();
                if (m & one) skeys[r] = v[i];
            }
        }
        // where this tile's items of bin `tid` go inside the segment
        S excl = 0;
        bool ok = true;
        if (q.ti == 0) {
            excl = digit.first(q.seg, q.sbase, ws2);
        } else if (tid < RADIX_BINS) {
            constexpr int LB = 4;
            const S* p = my - RADIX_BINS;
            int left = (int)q.ti;  // tiles before this one in the segment
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
        if (tid < RADIX_BINS) {
            if (ok) look_store(my, W::PREFIX | (excl + (S)total));
            goff[tid] = excl - (S)start;
        }
        if (__syncthreads_or(!ok)) {
            if (tid == 0) {
                atomicCAS(err, 0, ERR_WAIT_EXPIRED);
                atomicCAS(err, ERR_BAD_RUNS, ERR_WAIT_EXPIRED);
            }
            return;
        }
        // the next tile is claimed only now: a tile claimed while its CTA
        // still looks back would hold up everyone behind it
        if (tid == 0) next_tile = atomicAdd(claim, 1u);
        T* out = dst + q.sbase;
#pragma unroll 4
        for (int i = 0; i < IPT; ++i) {
            const int p = i * NT + tid;
            const T x = skeys[p];
            const S o = goff[digit(x)] + (S)p;
            // (o < slen always holds while the input does not change under the sort)
            if (p < q.cnt && o < (S)q.slen) out[o] = x;
        }
        __syncthreads();
    }
}

}  // namespace origami
