// Index arithmetic on CSR entries, for kernels and for host code that checks it.
#pragma once
#include <stdint.h>
#include <vector_types.h>

#if defined(__CUDACC__)
#define ACCX_EHD __host__ __device__ __forceinline__
#else
#define ACCX_EHD inline
#endif

// p[e0 .. e1) = x, a thread's chunk of at most N entries: 16-byte stores when it is whole
// (p 16-byte aligned, e0 a multiple of 4), and nothing outside the chunk.
template <int N>
ACCX_EHD void accx_fill_chunk(int32_t *p, uint32_t e0, uint32_t e1, int32_t x) {
  static_assert(N % 4 == 0, "whole 16-byte stores");
  if (e1 - e0 == N) {
    int4 q;
    q.x = q.y = q.z = q.w = x;
#if defined(__CUDACC__)
#pragma unroll
#endif
    for (int j = 0; j < N; j += 4) *reinterpret_cast<int4 *>(p + e0 + j) = q;
  } else {
    for (uint32_t e = e0; e < e1; e++) p[e] = x;
  }
}

// Positions are 32-bit and a CSR may have nearly 2^32 entries, so a position plus a step can
// wrap: these compare what is left instead.

// The end of a slice of `len` entries from e0 of a range that ends at `end` (e0 <= end).
ACCX_EHD uint32_t accx_slice_end(uint32_t e0, uint32_t len, uint32_t end) {
  return end - e0 > len ? e0 + len : end;
}
// The position `stride` after e in a loop over [.., end), e < end: `end` when there is none.
ACCX_EHD uint32_t accx_entry_step(uint32_t e, uint32_t stride, uint32_t end) { return accx_slice_end(e, stride, end); }
