// What the kernels that carry a state from token to token share.
#pragma once

#include "common.cuh"

__device__ __forceinline__ float log_sigmoid(float x) { return fminf(x, 0.f) - log1pf(expf(-fabsf(x))); }

// A step may hold decoded tokens beside portions of prompts.  The kernels for portions are then launched with their number,
// `portions`, and pass by the entries of one token, which state_step.cu takes from the step's list of them: neither kind's sums
// hang on the other's being there.  Without (0) all entries are taken, those of one token too.
__device__ __forceinline__ bool passed_by(int portions, int len) { return portions > 0 && len == 1; }

// The entry that block i of a launch over entries takes: number i, or the i-th of those that are not passed by; -1: none.
__device__ __forceinline__ int entry_of(int i, int portions, const int* __restrict__ cu_seqlens, int n_entries) {
  if (portions <= 0) return i;
  int begin = cu_seqlens[0];
  for (int e = 0; e < n_entries; ++e) {
    const int end = cu_seqlens[e + 1];
    if (end - begin != 1 && i-- == 0) return e;
    begin = end;
  }
  return -1;
}

// The token that item i of a launch over tokens is: number i, or that of entry work[2 i], which has one.
__device__ __forceinline__ int token_of(int i, const int* __restrict__ work, const int* __restrict__ cu_seqlens) {
  return work != nullptr ? cu_seqlens[work[2 * i]] : i;
}

// Segments of seg_len tokens that an entry has; one without tokens has one.
__device__ __forceinline__ int segments_of(int len, int seg_len, int portions) {
  return passed_by(portions, len) ? 0 : max(1, (len + seg_len - 1) / seg_len);
}

// Which entry and which of its segments the segment number g is; false if there is no such segment.  Segments are counted entry
// by entry; no lengths need to be known on the host, whose bound on their number is n / seg_len + entries.
__device__ __forceinline__ bool find_segment(const int* __restrict__ cu_seqlens, int n_entries, int seg_len, int portions, int g,
                                             int& entry, int& seg, int& n_seg) {
  int acc = 0;
  for (int e = 0; e < n_entries; ++e) {
    const int ns = segments_of(cu_seqlens[e + 1] - cu_seqlens[e], seg_len, portions);
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
