// What the kernels that carry a state from token to token share.
#pragma once

#include "common.cuh"

// Which entry and which of its segments the segment number g is; false if there is no such segment.  Segments of seg_len
// tokens are counted entry by entry (an entry without tokens has one); no lengths need to be known on the host, whose
// bound on their number is n / seg_len + entries.
__device__ __forceinline__ bool find_segment(const int* __restrict__ cu_seqlens, int n_entries, int seg_len, int g,
                                             int& entry, int& seg, int& n_seg) {
  int acc = 0;
  for (int e = 0; e < n_entries; ++e) {
    const int len = cu_seqlens[e + 1] - cu_seqlens[e];
    const int ns = max(1, (len + seg_len - 1) / seg_len);
    if (g < acc + ns) { entry = e; seg = g - acc; n_seg = ns; return true; }
    acc += ns;
  }
  return false;
}

__device__ __forceinline__ void cp_async_4(float* dst, const float* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_16(void* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// `bytes` (a multiple of 16) from global memory to shared memory, both on 16-byte boundaries; they count on `bar`.
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, int bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
               ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes), "r"((unsigned)__cvta_generic_to_shared(bar)) : "memory");
}
