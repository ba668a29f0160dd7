// Instantiation of the segmented bucket sort for uint64_t items.
#include "dispatch.h"
#include "seg_bucket_host.cuh"

namespace origami {

bool segbucket_fits_u64(uint64_t n, uint64_t nseg) { return SegBucketPlan<uint64_t>(n, nseg, n).fits(); }

uint64_t segbucket_scratch_bytes_u64(uint64_t n, uint64_t nseg) {
    return SegBucketScratch<uint64_t>(nullptr, SegBucketPlan<uint64_t>(n, nseg, n)).bytes;
}

cudaError_t segbucket_sort_u64(void* d, void* tmp, const uint64_t* off, uint64_t nseg, uint64_t n, uint64_t key_mask,
                               void* scratch, cudaStream_t st) {
    return segbucket_run<uint64_t>(static_cast<uint64_t*>(d), static_cast<uint64_t*>(tmp), off, nseg, n, key_mask, scratch, st);
}

void segbucket_behind(const SbBuffers<uint64_t>& buf, const SbGiven& given, const SbStarts& plain, const SegBucketPlan<uint64_t>& p,
                      uint64_t xin, uint64_t xout, const SegBucketScratch<uint64_t>& sc, cudaStream_t st) {
    segbucket_run<uint64_t>(buf, given, plain, p, xin, xout, sc, st);
}

void segbucket_prepare_u64() {
    SegBucketGrids<uint64_t, uint32_t>::get();
    SegBucketGrids<uint64_t, uint64_t>::get();
}

}  // namespace origami
