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
