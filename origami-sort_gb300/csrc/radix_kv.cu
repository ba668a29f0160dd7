// Instantiation of the radix passes for KV64 items.
#include "dispatch.h"
#include "radix_host.cuh"

namespace origami {

bool radix_fits_kv(uint64_t n, uint64_t sort_n) {
    if (!RadixPlan<KV64>::fits(n, sort_n)) return false;
    const RadixPlan<KV64> p(n, sort_n);
    return behind_plan(p, BucketPlan<KV64>(p)).fits();
}

uint64_t radix_scratch_bytes_kv(uint64_t n, uint64_t sort_n) { return radix_scratch_bytes<KV64>(n, sort_n); }

cudaError_t radix_sort_kv(void* d, void* tmp, uint64_t n, uint64_t sort_n, uint64_t key_mask, uint64_t out_mask, void* want,
                          void* scratch, cudaStream_t st) {
    return radix_sort<KV64>(static_cast<KV64*>(d), static_cast<KV64*>(tmp), n, sort_n, key_mask, out_mask, static_cast<KV64*>(want),
                          scratch, st);
}

bool one_bucket_kv(uint64_t n, uint64_t sort_n) { return one_bucket<KV64>(n, sort_n); }

cudaError_t bucket_one_kv(const void* d, void* want, uint64_t n, uint64_t key_mask, cudaStream_t st) {
    return bucket_one<KV64>(static_cast<const KV64*>(d), static_cast<KV64*>(want), n, key_mask, key_mask, nullptr, st);
}

}  // namespace origami
