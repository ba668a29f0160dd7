// Instantiation of the radix passes for uint64_t items.
#include "dispatch.h"
#include "radix_host.cuh"

namespace origami {

bool radix_fits_u64(uint64_t n, uint64_t sort_n) {
    if (!RadixPlan<uint64_t>::fits(n, sort_n)) return false;
    const RadixPlan<uint64_t> p(n, sort_n);
    return behind_plan(p, BucketPlan<uint64_t>(p)).fits();
}

uint64_t radix_scratch_bytes_u64(uint64_t n, uint64_t sort_n) { return radix_scratch_bytes<uint64_t>(n, sort_n); }

cudaError_t radix_sort_u64(void* d, void* tmp, uint64_t n, uint64_t sort_n, uint64_t key_mask, uint64_t out_mask, void* want,
                          void* scratch, cudaStream_t st) {
    return radix_sort<uint64_t>(static_cast<uint64_t*>(d), static_cast<uint64_t*>(tmp), n, sort_n, key_mask, out_mask, static_cast<uint64_t*>(want),
                          scratch, st);
}

bool one_bucket_u64(uint64_t n, uint64_t sort_n) { return one_bucket<uint64_t>(n, sort_n); }

cudaError_t bucket_one_u64(const void* d, void* want, uint64_t n, uint64_t key_mask, cudaStream_t st) {
    return bucket_one<uint64_t>(static_cast<const uint64_t*>(d), static_cast<uint64_t*>(want), n, key_mask, key_mask, nullptr, st);
}

}  // namespace origami
