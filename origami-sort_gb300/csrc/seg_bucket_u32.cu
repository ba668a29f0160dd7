// Instantiation of the segmented bucket sort for uint32_t items.
#include "dispatch.h"
#include "seg_bucket_host.cuh"

namespace origami {

bool segbucket_fits_u32(uint64_t n, uint64_t nseg) { return SegBucketPlan<uint32_t>(n, nseg, n).fits(); }

uint64_t segbucket_scratch_bytes_u32(uint64_t n, uint64_t nseg) {
    return SegBucketScratch<uint32_t>(nullptr, SegBucketPlan<uint32_t>(n, nseg, n)).bytes;
}

cudaError_t segbucket_sort_u32(void* d, void* tmp, const uint64_t* off, uint64_t nseg, uint64_t n, uint64_t key_mask,
                               void* scratch, cudaStream_t st) {
    return segbucket_run<uint32_t>(static_cast<uint32_t*>(d), static_cast<uint32_t*>(tmp), off, nseg, n, key_mask, scratch, st);
}

void segbucket_behind(const SbBuffers<uint32_t>& buf, const SbGiven& given, const SbStarts& plain, const SegBucketPlan<uint32_t>& p,
                      uint64_t xin, uint64_t xout, const SegBucketScratch<uint32_t>& sc, cudaStream_t st) {
    segbucket_run<uint32_t>(buf, given, plain, p, xin, xout, sc, st);
}

void segbucket_prepare_u32() {
    SegBucketGrids<uint32_t, uint32_t>::get();
    SegBucketGrids<uint32_t, uint64_t>::get();
}

}  // namespace origami
