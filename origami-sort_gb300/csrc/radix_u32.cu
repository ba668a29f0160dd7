// Instantiation of the radix passes for uint32_t items.
#include "dispatch.h"
#include "radix_host.cuh"

namespace origami {

bool radix_fits_u32(uint64_t n, uint64_t sort_n) { return RadixPlan<uint32_t>::fits(n, sort_n); }

uint64_t radix_scratch_bytes_u32(uint64_t n, uint64_t sort_n) { return radix_scratch_bytes<uint32_t>(n, sort_n); }

cudaError_t radix_sort_u32(void* d, void* tmp, uint64_t n, uint64_t sort_n, uint64_t key_mask, uint64_t out_mask, void* want,
                          void* scratch, cudaStream_t st) {
    return radix_sort<uint32_t>(static_cast<uint32_t*>(d), static_cast<uint32_t*>(tmp), n, sort_n, key_mask, out_mask, static_cast<uint32_t*>(want),
                          scratch, st);
}

bool one_bucket_u32(uint64_t n, uint64_t sort_n) { return one_bucket<uint32_t>(n, sort_n); }

cudaError_t bucket_one_u32(const void* d, void* want, uint64_t n, uint64_t key_mask, cudaStream_t st) {
    return bucket_one<uint32_t>(static_cast<const uint32_t*>(d), static_cast<uint32_t*>(want), n, key_mask, key_mask, nullptr, st);
}

}  // namespace origami
