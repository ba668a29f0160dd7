// Instantiation of the segmented bucket sort for KV64 items.
#include "dispatch.h"
#include "seg_bucket_host.cuh"

namespace origami {

bool segbucket_fits_kv(uint64_t n, uint64_t nseg) { return SegBucketPlan<KV64>(n, nseg, n).fits(); }

uint64_t segbucket_scratch_bytes_kv(uint64_t n, uint64_t nseg) {
    return SegBucketScratch<KV64>(nullptr, SegBucketPlan<KV64>(n, nseg, n)).bytes;
}

cudaError_t segbucket_sort_kv(void* d, void* tmp, const uint64_t* off, uint64_t nseg, uint64_t n, uint64_t key_mask,
                               void* scratch, cudaStream_t st) {
    return segbucket_run<KV64>(static_cast<KV64*>(d), static_cast<KV64*>(tmp), off, nseg, n, key_mask, scratch, st);
}

void segbucket_behind(const SbBuffers<KV64>& buf, const SbGiven& given, const SbStarts& plain, const SegBucketPlan<KV64>& p,
                      uint64_t xin, uint64_t xout, const SegBucketScratch<KV64>& sc, cudaStream_t st) {
    segbucket_run<KV64>(buf, given, plain, p, xin, xout, sc, st);
}

void segbucket_prepare_kv() {
    SegBucketGrids<KV64, uint32_t>::get();
    SegBucketGrids<KV64, uint64_t>::get();
}

}  // namespace origami
