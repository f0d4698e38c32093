// SCAN structural-clustering query on resident counts.
//
// Reference phases (scan-query-cuda/scan_xp_common.cu): similarity + core check
// (PostComputeCoreChecking :239-267), ClusterCore (:73-85) with the lock-free
// union-find of util/union_find.h:18-35, LabelNonCore/CheckHub (:87-111),
// PostProcess (:113-135), MarkClusterMinEleAsId (:137-158), PrepareResultOutput
// (:160-199) and Graph::Output (util/graph.cu:216-245).
//
// GPU form: one entry-parallel pass decides every similarity bit with the exact
// integer predicate (simpred.h) and counts similar entries per row with
// warp-aggregated atomics (the reference's core_count[u]++ is unsynchronised);
// union-find hooks the larger root under the smaller with atomicCAS, exactly as
// UnionThreadSafe does, so every component's root is its minimum id -- the
// cluster id MarkClusterMinEleAsId assigns; hubs keep the minimum and maximum
// root over core neighbours (two or more distinct roots iff min != max).
#include <cub/cub.cuh>

#include <algorithm>
#include <mutex>
#include <string>
#include <vector>

#include "accx_internal.h"
#include "devutil.cuh"
#include "entries.h"
#include "simpred.h"

// query counters
#define Q_SIMILAR 0
#define Q_CORES 1
#define Q_CLUSTERS 2
#define Q_HUBS 3
#define Q_OUTLIERS 4
#define Q_PAIRS 5
#define Q_DIGEST 6
#define Q_BIG 7
#define Q_CORELIST 8   // cores with short rows, in the core list
#define Q_PUSH 9       // slices of the other cores' rows, and those cores times Q_LONG
#define Q_LONG (1ull << 40)
#define Q_NUM 10

__device__ __forceinline__ unsigned long long accx_mix64_dev(unsigned long long x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

// The float nearest to c^2 / (du dv) but for rare last-bit ties (error below 2^-24
// (1 + 2^-20) relative), by Dekker's division of double-length numbers (Numerische Mathematik
// 18, 1971): each product as an unevaluated pair of floats (exact by a fused multiply-add),
// the quotient of their leading parts, and one correction by the remainder.  FP64 and conversions of 64-bit integers run
// at a small fraction of the FP32 rate here: the keys of 128M entries took 3.27 ms with
// FP64 division and 1.32 ms through 64-bit integers; now 0.90.  Operands of 2^24 and more
// (no float holds them exactly) take the 64-bit way.
__device__ __noinline__ float accx_ratio_wide(uint32_t c, uint32_t du, uint32_t dv) {
  const unsigned long long a = (unsigned long long)c * c, d = (unsigned long long)du * dv;
  const float ah = __ull2float_rn(a), dh = __ull2float_rn(d);
  // |a - ah| < 2^40, exact as a signed difference (mod 2^64: ah may round up to 2^64)
  const float al = __ll2float_rn((long long)(a - (ah >= 18446744073709551616.0f ? 0ull : (unsigned long long)ah)));
  const float dl = __ll2float_rn((long long)(d - (dh >= 18446744073709551616.0f ? 0ull : (unsigned long long)dh)));
  const float q = __fdiv_rn(ah, dh);
  const float r = __fmaf_rn(-q, dl, __fmaf_rn(-q, dh, ah) + al);
  return __fadd_rn(q, __fdividef(r, dh));
}
__device__ __forceinline__ float accx_ratio(uint32_t c, uint32_t du, uint32_t dv) {
  if ((c | du | dv) >> 24) return accx_ratio_wide(c, du, dv);
  const float cf = __uint2float_rn(c), uf = __uint2float_rn(du), vf = __uint2float_rn(dv);
  const float ah = __fmul_rn(cf, cf), al = __fmaf_rn(cf, cf, -ah), dh = __fmul_rn(uf, vf), dl = __fmaf_rn(uf, vf, -dh);
  const float i = __fdividef(1.f, dh), q = __fmul_rn(ah, i);
  const float r = __fmaf_rn(-q, dl, __fmaf_rn(-q, dh, ah) + al);
  return __fmaf_rn(r, i, q);
}

// Per-entry similarity key, built once after each count: the float nearest to
// x^2 = cnn^2 / (du * dv).  A query compares it with the squared threshold M^2
// of its eps; only keys within 2^-21 (relative) of M^2 -- where float rounding
// could matter -- take the exact-integer test (simpred.h) with cnn, du, dv read
// back from the graph.
// A thread takes eight consecutive entries: one row search inside their 256-entry tile
// (tilerow), the neighbours' offsets gathered together.
__global__ void __launch_bounds__(256) k_simkey(const uint32_t *__restrict__ off, const uint32_t *__restrict__ tilerow,
                                                const int32_t *__restrict__ dst, const int32_t *__restrict__ cnt,
                                                uint32_t m, int32_t bias, float *__restrict__ key,
                                                uint32_t *__restrict__ src) {
  const uint32_t nb = m / 8 + (m % 8 ? 1 : 0);
  for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < nb; c += gridDim.x * blockDim.x) {
    const uint32_t e0 = c * 8, k = min(m - e0, 8u), t = e0 / 256u;
    uint32_t v[8], n[8], dv[8];
    if (k == 8) {
      const int4 a = __ldg(reinterpret_cast<const int4 *>(dst + e0)), b = __ldg(reinterpret_cast<const int4 *>(dst + e0) + 1);
      const int4 p = __ldg(reinterpret_cast<const int4 *>(cnt + e0)), q = __ldg(reinterpret_cast<const int4 *>(cnt + e0) + 1);
      v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
      n[0] = p.x; n[1] = p.y; n[2] = p.z; n[3] = p.w; n[4] = q.x; n[5] = q.y; n[6] = q.z; n[7] = q.w;
    } else {
#pragma unroll
      for (int i = 0; i < 8; i++) {
        v[i] = (uint32_t)i < k ? (uint32_t)__ldg(dst + e0 + i) : 0u;
        n[i] = (uint32_t)i < k ? (uint32_t)__ldg(cnt + e0 + i) : 0u;
      }
    }
#pragma unroll
    for (int i = 0; i < 8; i++) dv[i] = __ldg(off + v[i] + 1) - __ldg(off + v[i]) + 1;
    uint32_t u = accx_row_of(off, __ldg(tilerow + t), __ldg(tilerow + t + 1) + 1, e0);
    uint32_t re = __ldg(off + u + 1), du = re - __ldg(off + u) + 1;
    float x[8];
    uint32_t r[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      while ((uint32_t)i < k && re <= e0 + i) {  // the next non-empty row
        const uint32_t rb = re;
        u++;
        re = __ldg(off + u + 1);
        du = re - rb + 1;
      }
      x[i] = accx_ratio((uint32_t)((int32_t)n[i] - bias + 2), du, dv[i]);
      r[i] = u;
    }
    if (k == 8) {
      reinterpret_cast<float4 *>(key + e0)[0] = make_float4(x[0], x[1], x[2], x[3]);
      reinterpret_cast<float4 *>(key + e0)[1] = make_float4(x[4], x[5], x[6], x[7]);
      reinterpret_cast<uint4 *>(src + e0)[0] = make_uint4(r[0], r[1], r[2], r[3]);
      reinterpret_cast<uint4 *>(src + e0)[1] = make_uint4(r[4], r[5], r[6], r[7]);
    } else {
      for (uint32_t i = 0; i < k; i++) {
        key[e0 + i] = x[i];
        src[e0 + i] = r[i];
      }
    }
  }
}

// Similarity bits from the keys: a streaming pass, eight entries a thread (two 16-byte
// loads, one byte of the bit array), and in the same pass the caller's 0/1 bytes when
// wanted (out, 8-byte aligned).  Bound by HBM: 4 bytes read an entry.  128M entries: 452
// us with one entry a thread and a ballot, plus 189 for the bytes in a pass of their own; now
// 125 for both (5.1 TB/s).
__global__ void __launch_bounds__(256) k_sim_keys(const float *__restrict__ key, const uint32_t *__restrict__ off,
                                                  const uint32_t *__restrict__ src, const int32_t *__restrict__ dst,
                                                  const int32_t *__restrict__ cnt, uint32_t m, int32_t bias,
                                                  accx_simq q, float lo, float hi, uint8_t *__restrict__ simbits,
                                                  uint8_t *__restrict__ out, unsigned long long *__restrict__ qc) {
  const uint32_t stride = gridDim.x * blockDim.x;
  const uint32_t nb = ((m + 31) / 32) * 4;  // bytes of whole words: bits past m are zero
  uint32_t similar = 0;
  for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < nb; c += stride) {
    const uint32_t e0 = c * 8;
    uint32_t bits = 0;
    if (e0 < m) {
      const uint32_t valid = m - e0 >= 8 ? 0xffu : (1u << (m - e0)) - 1u;
      if (q.mode != 0) {
        bits = q.mode == 1 ? 0xffu : 0u;
      } else {
        float k[8];
        if (valid == 0xffu) {
          const float4 a = __ldg(reinterpret_cast<const float4 *>(key + e0));
          const float4 b = __ldg(reinterpret_cast<const float4 *>(key + e0) + 1);
          k[0] = a.x; k[1] = a.y; k[2] = a.z; k[3] = a.w;
          k[4] = b.x; k[5] = b.y; k[6] = b.z; k[7] = b.w;
        } else {
#pragma unroll
          for (int i = 0; i < 8; i++) k[i] = (valid >> i) & 1u ? __ldg(key + e0 + i) : -1.f;
        }
        uint32_t band = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) {
          bits |= (k[i] > hi ? 1u : 0u) << i;
          band |= (k[i] >= lo && k[i] <= hi ? 1u : 0u) << i;
        }
        for (band &= valid; band; band &= band - 1) {
          // ambiguous band (exact ties x == eps land here): exact test with the entry's
          // own numbers
          const uint32_t i = __ffs(band) - 1, e = e0 + i, u = __ldg(src + e), v = (uint32_t)dst[e];
          if (accx_similar(q, (uint32_t)(cnt[e] - bias + 2), off[u + 1] - off[u] + 1, off[v + 1] - off[v] + 1))
            bits |= 1u << i;
        }
      }
      bits &= valid;
      if (out) {
        // four bits to four 0/1 bytes: copies shifted by 7, 14 and 21 put bit i at byte i
        const uint2 y = make_uint2(((bits & 15u) * 0x00204081u) & 0x01010101u, ((bits >> 4) * 0x00204081u) & 0x01010101u);
        if (valid == 0xffu) {
          *reinterpret_cast<uint2 *>(out + e0) = y;
        } else {
          for (uint32_t i = 0; e0 + i < m; i++) out[e0 + i] = (uint8_t)((bits >> i) & 1u);
        }
      }
    }
    simbits[c] = (uint8_t)bits;
    similar += __popc(bits);
  }
  similar = __reduce_add_sync(ACCX_FULL_MASK, similar);
  if ((threadIdx.x & 31) == 0 && similar) atomicAdd(&qc[Q_SIMILAR], (unsigned long long)similar);
}

// Cores from the similarity bits: core_count[u] = popcount of row u's bits.
// One thread per vertex, four words' loads in flight (a warp for each row above 256
// entries measured slower: hubs' ids lie together); rows above BIG_ROW by a CTA
// (k_cores_big).  Also resets labels, union-find roots
// and hub ranges, writes the core bitmap (n/8 bytes, kept in L2 for the random lookups
// that follow), and lists the cores for k_hub_push: short rows as vertices, longer ones
// as slices.
#define BIG_ROW 4096
#define PUSH_ROW 256u     // cores with rows up to this are one warp's work
#define PUSH_SLICE 512u   // entries of a longer core row a warp pushes
#define CORE_KEEP 64u     // groups of 32 vertices with listed cores a warp gathers before one atomic places them
__device__ __forceinline__ uint32_t accx_row_word(const uint32_t *__restrict__ bits, uint32_t w, uint32_t b,
                                                  uint32_t e) {
  uint32_t x = __ldg(bits + w);
  if (w == b >> 5) x &= 0xffffffffu << (b & 31);
  if (w == (e - 1) >> 5 && (e & 31)) x &= 0xffffffffu >> (32 - (e & 31));
  return __popc(x);
}

__device__ __forceinline__ void accx_push_slices(uint32_t u, uint32_t deg, uint2 *__restrict__ push,
                                                 unsigned long long *__restrict__ qc) {
  const uint32_t ns = (deg + PUSH_SLICE - 1) / PUSH_SLICE;
  const unsigned long long p = atomicAdd(&qc[Q_PUSH], Q_LONG + ns) % Q_LONG;
  for (uint32_t j = 0; j < ns; j++) push[p + j] = make_uint2(u, j);
}

__global__ void __launch_bounds__(256) k_cores(const uint32_t *__restrict__ off, uint32_t n, int mu,
                                               const uint32_t *__restrict__ simbits, int32_t *__restrict__ label,
                                               int32_t *__restrict__ parent, int32_t *__restrict__ hubmin,
                                               int32_t *__restrict__ hubmax, uint32_t *__restrict__ corebits,
                                               uint32_t *__restrict__ big, uint32_t *__restrict__ corelist,
                                               uint2 *__restrict__ push, unsigned long long *__restrict__ qc) {
  __shared__ uint2 s_keep[8][CORE_KEEP];  // first vertex and which of its 32
  uint2 *keep = s_keep[threadIdx.x >> 5];
  uint32_t groups = 0, kept = 0;
  const uint32_t stride = gridDim.x * blockDim.x;  // a multiple of 32
  const int lane = threadIdx.x & 31;
  auto flush = [&]() {
    __syncwarp();
    unsigned long long p = 0;
    if (lane == 0) p = atomicAdd(&qc[Q_CORELIST], (unsigned long long)kept);
    p = __shfl_sync(ACCX_FULL_MASK, p, 0);
    for (uint32_t i = 0; i < groups; i++) {
      const uint2 g = keep[i];
      if ((g.y >> lane) & 1u) corelist[p + __popc(g.y & ((1u << lane) - 1u))] = g.x + lane;
      p += __popc(g.y);
    }
    __syncwarp();
    groups = kept = 0;
  };
  for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < ((n + 31) & ~31u); u += stride) {
    uint32_t b = 0, e = 0, c = 0;
    if (u < n) {
      b = __ldg(off + u);
      e = __ldg(off + u + 1);
      parent[u] = (int32_t)u;
      hubmin[u] = 0x7fffffff;
      hubmax[u] = -1;
    }
    const uint32_t deg = e - b;
    const bool is_big = deg > BIG_ROW;
    if (deg && !is_big)
      for (uint32_t w = b >> 5, w1 = (e - 1) >> 5; w <= w1; w += 4) {
        uint32_t t[4];
#pragma unroll
        for (int i = 0; i < 4; i++) t[i] = w + i <= w1 ? accx_row_word(simbits, w + i, b, e) : 0u;
        c += t[0] + t[1] + t[2] + t[3];
      }
    const bool core = u < n && !is_big && (int)c >= mu;
    if (is_big) big[atomicAdd(&qc[Q_BIG], 1ull)] = u;  // decided by k_cores_big
    else if (u < n) label[u] = core ? ACCX_CORE : ACCX_UNCLASSIFIED;
    const unsigned w = __ballot_sync(ACCX_FULL_MASK, core);
    if (lane == 0 && u < n) corebits[u >> 5] = w;
    const bool brief = core && deg <= PUSH_ROW;
    const unsigned bw = __ballot_sync(ACCX_FULL_MASK, brief);
    if (bw) {
      if (lane == 0) keep[groups] = make_uint2(u, bw);
      kept += __popc(bw);
      if (++groups == CORE_KEEP) flush();
    }
    if (core && !brief) accx_push_slices(u, deg, push, qc);
  }
  if (groups) flush();
}

__global__ void __launch_bounds__(256) k_cores_big(const uint32_t *__restrict__ off, int mu,
                                                   const uint32_t *__restrict__ simbits, const uint32_t *__restrict__ big,
                                                   int32_t *__restrict__ label, uint32_t *__restrict__ corebits,
                                                   uint2 *__restrict__ push, unsigned long long *__restrict__ qc) {
  __shared__ uint32_t part[8];
  const unsigned long long nb = qc[Q_BIG];
  for (unsigned long long i = blockIdx.x; i < nb; i += gridDim.x) {
    const uint32_t u = big[i], b = off[u], e = off[u + 1];
    uint32_t c = 0;
    for (uint32_t w = (b >> 5) + threadIdx.x; w <= (e - 1) >> 5; w += blockDim.x) c += accx_row_word(simbits, w, b, e);
    c = __reduce_add_sync(ACCX_FULL_MASK, c);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t t = 0;
      for (int k = 0; k < (int)(blockDim.x >> 5); k++) t += part[k];
      const bool core = (int)t >= mu;
      label[u] = core ? ACCX_CORE : ACCX_UNCLASSIFIED;
      if (core) {
        atomicOr(&corebits[u >> 5], 1u << (u & 31));
        accx_push_slices(u, e - b, push, qc);
      }
    }
    __syncthreads();
  }
}

__device__ __forceinline__ bool accx_is_core(const uint32_t *__restrict__ corebits, uint32_t v) {
  return (__ldg(corebits + (v >> 5)) >> (v & 31)) & 1u;
}

// Root with path halving; parents only ever point to smaller ids.
__device__ __forceinline__ int32_t uf_find(volatile int32_t *parent, int32_t x) {
  int32_t cur = parent[x];
  if (cur != x) {
    int32_t prev = x, next;
    while (cur > (next = parent[cur])) {
      parent[prev] = next;
      prev = cur;
      cur = next;
    }
  }
  return cur;
}

// Union of two cores' components.  UnionThreadSafe (union_find.h:22-35): hook the larger
// root under the smaller.
__device__ __forceinline__ void uf_unite(volatile int32_t *vp, int32_t *parent, uint32_t u, uint32_t v) {
  for (;;) {
    int32_t ru = uf_find(vp, (int32_t)u), rv = uf_find(vp, (int32_t)v);
    if (ru == rv) break;
    int32_t lo = ru < rv ? ru : rv, hi = ru < rv ? rv : ru;
    if (atomicCAS(&parent[hi], hi, lo) == hi) break;
  }
}

// Union over similar core-core entries, in one of two forms; a kernel returns at once when
// the query is not its own.
// hook_words, few similar entries a core (below HOOK_DENSE): a thread a word of the similarity
// bits, whose entries are mostly one row's and are united one after another.  There is little
// to fight over.  On graphs of HOOK_OWN entries and more it is a kernel of its own, which has the
// L1 to itself (with the other form's shared memory a ring of 16 entries a vertex took 714
// us, without 576); on smaller ones the launch costs more (2 us) than that.
// By lanes, many: a warp takes 32 words, gathers the entries of their set bits in shared
// memory and gives every lane one entry (an entry is a chain of dependent random reads: a
// thread working off a word's bits alone left most of the machine waiting).  A first pass
// (FIRST) lowers cores' parents to their smallest similar core neighbour, one atomic minimum
// an entry, nothing to wait for or to retry.  It loses links, but the second unites over
// every entry again and finds nearly all of them done, where without it the cores of one big
// cluster fight over the same roots.  An eighth of the vertices, by a hash, stay out of the
// first pass: where ids follow the graph's layout (a ring, a lattice) the minima would make
// chains of many thousands of links that the second has to walk.
// The whole union, us, by lanes / by words: R-MAT 22 50 / 176, R-MAT 16 with 64 edges a
// vertex 58 / 204, cliques of 1500 91 / 334; Erdos-Renyi 2M with 6 similar entries a core
// 1350 / 666, power law 1M 546 / 145, ring of 16 entries a vertex 1170 / 576, cliques of 20
// 56 / 58.
#define HOOK_WARPS 8
#define HOOK_DENSE 32ull
__device__ __forceinline__ int hook_kind(const unsigned long long *__restrict__ qc) {  // 0: nothing to unite
  const unsigned long long cores = qc[Q_CORELIST] + qc[Q_PUSH] / Q_LONG;
  return cores < 2 ? 0 : qc[Q_SIMILAR] < HOOK_DENSE * cores ? 1 : 2;
}
#define HOOK_OWN (1u << 22)
__device__ __forceinline__ void hook_words(const uint32_t *__restrict__ src, const int32_t *__restrict__ dst, uint32_t m,
                                           const uint32_t *__restrict__ simbits,
                                           const uint32_t *__restrict__ corebits, int32_t *parent) {
  volatile int32_t *vp = parent;
  const uint32_t words = (m + 31) / 32;
  for (uint32_t wi = blockIdx.x * blockDim.x + threadIdx.x; wi < words; wi += gridDim.x * blockDim.x)
    for (uint32_t w = __ldg(simbits + wi); w; w &= w - 1) {
      const uint32_t e = wi * 32u + (uint32_t)(__ffs(w) - 1), v = (uint32_t)__ldg(dst + e);
      if (!accx_is_core(corebits, v)) continue;
      const uint32_t u = __ldg(src + e);
      if (u < v && accx_is_core(corebits, u)) uf_unite(vp, parent, u, v);
    }
}
__global__ void __launch_bounds__(HOOK_WARPS * 32) k_hook_words(const uint32_t *__restrict__ src,
                                                                const int32_t *__restrict__ dst, uint32_t m,
                                                                const uint32_t *__restrict__ simbits,
                                                                const uint32_t *__restrict__ corebits,
                                                                const unsigned long long *__restrict__ qc,
                                                                int32_t *parent) {
  if (hook_kind(qc) == 1) hook_words(src, dst, m, simbits, corebits, parent);
}
template <bool FIRST>
__global__ void __launch_bounds__(HOOK_WARPS * 32) k_hook_lanes(const uint32_t *__restrict__ src,
                                                                const int32_t *__restrict__ dst, uint32_t m,
                                                                const uint32_t *__restrict__ simbits,
                                                                const uint32_t *__restrict__ corebits,
                                                                const unsigned long long *__restrict__ qc,
                                                                int32_t *parent) {
  __shared__ uint16_t s_q[HOOK_WARPS][1024];  // places in the warp's 32 words
  const int kind = hook_kind(qc);
  if (FIRST && kind == 1 && m < HOOK_OWN) hook_words(src, dst, m, simbits, corebits, parent);
  if (kind != 2) return;
  volatile int32_t *vp = parent;
  const int lane = threadIdx.x & 31;
  uint16_t *q = s_q[threadIdx.x >> 5];
  const uint32_t words = (m + 31) / 32, nw = gridDim.x * HOOK_WARPS;
  for (unsigned long long w0 = 32ull * (blockIdx.x * HOOK_WARPS + (threadIdx.x >> 5)); w0 < words; w0 += 32ull * nw) {
    const uint32_t wi = (uint32_t)w0 + lane;
    uint32_t w = wi < words ? __ldg(simbits + wi) : 0u;
    uint32_t at = __popc(w);
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t a = __shfl_up_sync(ACCX_FULL_MASK, at, d);
      if (lane >= d) at += a;
    }
    const uint32_t total = __shfl_sync(ACCX_FULL_MASK, at, 31);
    at -= __popc(w);
    for (; w; w &= w - 1) q[at++] = (uint16_t)(lane * 32 + __ffs(w) - 1);
    __syncwarp();
    for (uint32_t i = lane; i < total; i += 32) {
      const uint32_t e = (uint32_t)w0 * 32u + q[i], u = __ldg(src + e), v = (uint32_t)__ldg(dst + e);
      if (u >= v || !accx_is_core(corebits, v) || !accx_is_core(corebits, u)) continue;
      if (!FIRST) uf_unite(vp, parent, u, v);
      else if ((v * 0x9E3779B1u) >> 29) atomicMin(&parent[v], (int32_t)u);
    }
    __syncwarp();
  }
}

// Every core's parent to its root.  Other threads shorten the same paths: all writes are
// minima, so that one with an ancestor read earlier never undoes a root written since (with
// plain stores a core could keep an ancestor for its cluster).
__global__ void k_compress(uint32_t n, const uint32_t *__restrict__ corebits, int32_t *parent) {
  volatile int32_t *vp = parent;
  for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < n; u += gridDim.x * blockDim.x) {
    if (!accx_is_core(corebits, u)) continue;
    int32_t prev = (int32_t)u, cur = vp[u], next;
    while (cur > (next = vp[cur])) {
      atomicMin(&parent[prev], next);
      prev = cur;
      cur = next;
    }
    atomicMin(&parent[u], cur);
  }
}

// Hubs, pushed from the core side: core vertex v streams N(v) and folds its cluster root
// into the [min, max] range of every non-core neighbour (CheckHub ignores similarity: any
// core neighbour counts).  A warp per listed core with a short row, or per slice of a
// longer row: walking the core bitmap instead, one warp had all the cores of a word,
// whose rows can be hubs' (R-MAT 13: 86 us, now 8; R-MAT 22, with a grid of CTAs for the
// longest rows: 97, now 70).  Where a warp has HUB_PACK listed cores and more, it takes 32 at a
// time and streams their rows as one (a lattice of 6M cores with four entries each
// 777 us with a row a step).
#define HUB_PACK 16u
__device__ __forceinline__ void accx_hub_credit(uint32_t u, int32_t r, const uint32_t *__restrict__ corebits,
                                                int32_t *__restrict__ hubmin, int32_t *__restrict__ hubmax) {
  if (u == 0xffffffffu || accx_is_core(corebits, u)) return;
  atomicMin(&hubmin[u], r);
  atomicMax(&hubmax[u], r);
}
__device__ __forceinline__ void accx_hub_range(const int32_t *__restrict__ dst, uint32_t b, uint32_t e, int32_t r,
                                               int lane, const uint32_t *__restrict__ corebits,
                                               int32_t *__restrict__ hubmin, int32_t *__restrict__ hubmax) {
  const uint32_t len = e - b;
  for (uint32_t i0 = 0; i0 < len; i0 += 128) {
    uint32_t u[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint32_t i = i0 + 32 * k + lane;
      u[k] = i < len ? (uint32_t)__ldg(dst + b + i) : 0xffffffffu;
    }
#pragma unroll
    for (int k = 0; k < 4; k++) accx_hub_credit(u[k], r, corebits, hubmin, hubmax);
  }
}
__global__ void __launch_bounds__(256) k_hub_push(const uint32_t *__restrict__ off, const int32_t *__restrict__ dst,
                                                  const uint32_t *__restrict__ corelist, const uint2 *__restrict__ push,
                                                  const unsigned long long *__restrict__ qc,
                                                  const uint32_t *__restrict__ corebits,
                                                  const int32_t *__restrict__ parent, int32_t *__restrict__ hubmin,
                                                  int32_t *__restrict__ hubmax) {
  // the rows of 32 cores: where each begins in their concatenation, less its place in dst
  __shared__ uint32_t s_pre[8][32], s_beg[8][32];
  __shared__ int32_t s_root[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned long long nw = (gridDim.x * blockDim.x) >> 5, w0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const unsigned long long np = qc[Q_PUSH] % Q_LONG, nc = qc[Q_CORELIST];
  for (unsigned long long i = w0; i < np; i += nw) {
    const uint2 it = __ldg(push + i);
    const uint32_t b = __ldg(off + it.x) + it.y * PUSH_SLICE, e = accx_slice_end(b, PUSH_SLICE, __ldg(off + it.x + 1));
    accx_hub_range(dst, b, e, parent[it.x], lane, corebits, hubmin, hubmax);
  }
  if (nc < HUB_PACK * nw) {
    for (unsigned long long i = w0; i < nc; i += nw) {
      const uint32_t v = __ldg(corelist + i);
      accx_hub_range(dst, __ldg(off + v), __ldg(off + v + 1), parent[v], lane, corebits, hubmin, hubmax);
    }
    return;
  }
  uint32_t *pre = s_pre[warp], *beg = s_beg[warp];
  int32_t *root = s_root[warp];
  for (unsigned long long i = 32 * w0; i < nc; i += 32 * nw) {
    uint32_t b = 0, len = 0;
    if (i + lane < nc) {
      const uint32_t v = __ldg(corelist + i + lane);
      b = __ldg(off + v);
      len = __ldg(off + v + 1) - b;
      root[lane] = parent[v];
    }
    uint32_t incl = len;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t a = __shfl_up_sync(ACCX_FULL_MASK, incl, d);
      if (lane >= d) incl += a;
    }
    const uint32_t tot = __shfl_sync(ACCX_FULL_MASK, incl, 31);
    pre[lane] = incl - len;  // an empty row begins where the next one does
    beg[lane] = b;
    __syncwarp();
    for (uint32_t c0 = 0; c0 < tot; c0 += 128) {
      uint32_t u[4], s[4];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const uint32_t c = c0 + 32 * k + lane;
        // the last row that begins at or before c
        uint32_t j = 0;
#pragma unroll
        for (int d = 16; d >= 1; d >>= 1) j += pre[j + d] <= c ? d : 0;
        s[k] = j;
        u[k] = c < tot ? (uint32_t)__ldg(dst + beg[j] + (c - pre[j])) : 0xffffffffu;
      }
#pragma unroll
      for (int k = 0; k < 4; k++) accx_hub_credit(u[k], root[s[k]], corebits, hubmin, hubmax);
    }
    __syncwarp();
  }
}

__global__ void k_finish(uint32_t n, int32_t *__restrict__ label, const int32_t *__restrict__ parent,
                         const int32_t *hubmin, const int32_t *__restrict__ hubmax,
                         int32_t *cluster_out, unsigned long long *__restrict__ qc) {  // cluster_out may be hubmin
  unsigned long long cores = 0, clusters = 0, hubs = 0, outl = 0, dig = 0;
  for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < n; u += gridDim.x * blockDim.x) {
    int32_t l = label[u];
    if (l == ACCX_CORE) {
      cores++;
      if (parent[u] == (int32_t)u) clusters++;
    } else if (hubmax[u] >= 0 && hubmin[u] != hubmax[u]) {
      label[u] = ACCX_HUB;
      l = ACCX_HUB;
      hubs++;
    } else {
      outl++;
    }
    const int32_t cl = (l == ACCX_CORE) ? parent[u] : -1;
    if (cluster_out) cluster_out[u] = cl;
    dig += accx_mix64_dev(((unsigned long long)u << 34) ^ ((unsigned long long)(uint32_t)l << 32) ^ (uint32_t)cl);
  }
  cores = __reduce_add_sync(ACCX_FULL_MASK, (unsigned)cores);
  clusters = __reduce_add_sync(ACCX_FULL_MASK, (unsigned)clusters);
  hubs = __reduce_add_sync(ACCX_FULL_MASK, (unsigned)hubs);
  outl = __reduce_add_sync(ACCX_FULL_MASK, (unsigned)outl);
  for (int d = 16; d >= 1; d >>= 1) dig += __shfl_xor_sync(ACCX_FULL_MASK, dig, d);
  if ((threadIdx.x & 31) == 0) {
    if (dig) atomicAdd(&qc[Q_DIGEST], dig);
    if (cores) atomicAdd(&qc[Q_CORES], cores);
    if (clusters) atomicAdd(&qc[Q_CLUSTERS], clusters);
    if (hubs) atomicAdd(&qc[Q_HUBS], hubs);
    if (outl) atomicAdd(&qc[Q_OUTLIERS], outl);
  }
}

__global__ void k_bits_to_bytes(const uint32_t *__restrict__ bits, uint32_t m, uint8_t *__restrict__ out) {
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < m; e = accx_entry_step(e, stride, m))
    out[e] = (bits[e >> 5] >> (e & 31)) & 1u;
}

// (cluster id, non-core vertex) keys for core u, non-core v, similar (u,v).
template <int TILE>
__global__ void __launch_bounds__(TILE) k_pairs(const uint32_t *__restrict__ off, const uint32_t *__restrict__ tilerow, const int32_t *__restrict__ dst,
                                                uint32_t n, uint32_t m, const uint32_t *__restrict__ simbits,
                                                const int32_t *__restrict__ label, const int32_t *__restrict__ parent,
                                                unsigned long long *__restrict__ keys, unsigned long long cap,
                                                unsigned long long *__restrict__ qc) {
  __shared__ accx_tile_rows<TILE> sh;
  uint32_t base = blockIdx.x * (uint32_t)TILE;
  uint32_t e = base + threadIdx.x;
  uint32_t u = accx_tile_row<TILE>(off, tilerow, n, m, base, e, &sh);
  bool act = false;
  unsigned long long key = 0;
  if (e < m && ((simbits[e >> 5] >> (e & 31)) & 1u) && label[u] == ACCX_CORE) {
    uint32_t v = (uint32_t)dst[e];
    if (label[v] != ACCX_CORE) {
      act = true;
      key = ((unsigned long long)(uint32_t)parent[u] << 32) | v;
    }
  }
  unsigned mask = __ballot_sync(ACCX_FULL_MASK, act);
  if (!mask) return;
  int lane = threadIdx.x & 31, leader = __ffs(mask) - 1;
  unsigned long long p = 0;
  if (lane == leader) p = atomicAdd(&qc[Q_PAIRS], (unsigned long long)__popc(mask));
  p = __shfl_sync(ACCX_FULL_MASK, p, leader);
  if (act && keys) {
    unsigned long long idx = p + __popc(mask & ((1u << lane) - 1u));
    if (idx < cap) keys[idx] = key;
  }
}

void accx_query_ctx_release(accx_query_ctx *q) {
  void *ptrs[] = {q->d_simbits, q->d_corelist,  q->d_label, q->d_parent,    q->d_hubmin,   q->d_hubmax,
                  q->d_push,    q->d_qcounters, q->d_pairs, q->d_pairs_tmp, q->d_corebits, q->d_big};
  accx_dev_free_all(ptrs, (int)(sizeof(ptrs) / sizeof(ptrs[0])), nullptr);
  *q = accx_query_ctx();
}

// A temporary of the pool, freed on its stream on every way out of a call.
struct stream_block {
  void *p = nullptr;
  cudaStream_t s;
  explicit stream_block(cudaStream_t st) : s(st) {}
  ~stream_block() {
    if (p) cudaFreeAsync(p, s);
  }
  stream_block(const stream_block &) = delete;
  stream_block &operator=(const stream_block &) = delete;
};

static int ensure_query_arrays(const accx_graph *g, accx_query_ctx *q) {
  if (q->d_simbits && (q->n != g->n || q->m != g->m)) return ACCX_ERR_INVALID_ARG;  // made for another graph
  accx_graph *gm = const_cast<accx_graph *>(g);  // which may give scratch back
  q->n = g->n;
  q->m = g->m;
  if (q->d_big) return ACCX_OK;  // the last of them
  const size_t n = g->n ? g->n : 1, words = (g->m + 31) / 32 + 1;
  if (!q->d_simbits) ACCX_CUDA_TRY(accx_graph_alloc(gm, (void **)&q->d_simbits, sizeof(uint32_t) * words, nullptr));
  if (!q->d_corelist) ACCX_CUDA_TRY(accx_graph_alloc(gm, (void **)&q->d_corelist, sizeof(uint32_t) * n, nullptr));
  // rows above PUSH_ROW have at most 1 + degree/PUSH_SLICE slices
  if (!q->d_push) ACCX_CUDA_TRY(accx_graph_alloc(gm, (void **)&q->d_push, sizeof(uint2) * (g->m / PUSH_ROW + g->m / PUSH_SLICE + 2), nullptr));
  if (!q->d_label) ACCX_CUDA_TRY(accx_graph_alloc(gm, (void **)&q->d_label, sizeof(int32_t) * n, nullptr));
  if (!q->d_parent) ACCX_CUDA_TRY(accx_graph_alloc(gm, (void **)&q->d_parent, sizeof(int32_t) * n, nullptr));
  if (!q->d_hubmin) ACCX_CUDA_TRY(accx_graph_alloc(gm, (void **)&q->d_hubmin, sizeof(int32_t) * n, nullptr));
  if (!q->d_hubmax) ACCX_CUDA_TRY(accx_graph_alloc(gm, (void **)&q->d_hubmax, sizeof(int32_t) * n, nullptr));
  if (!q->d_qcounters) ACCX_CUDA_TRY(accx_graph_alloc(gm, (void **)&q->d_qcounters, sizeof(unsigned long long) * Q_NUM, nullptr));
  if (!q->d_corebits) ACCX_CUDA_TRY(accx_graph_alloc(gm, (void **)&q->d_corebits, sizeof(uint32_t) * (n / 32 + 2), nullptr));
  if (!q->d_big) ACCX_CUDA_TRY(accx_graph_alloc(gm, (void **)&q->d_big, sizeof(uint32_t) * (g->m / BIG_ROW + 2), nullptr));
  ACCX_CUDA_TRY(accx_dev_wait(nullptr));
  return ACCX_OK;
}

extern "C" int accx_scan_query_ctx(const accx_graph *g, accx_query_ctx *q, double eps, int mu, uint8_t *sim,
                                   int32_t *label, int32_t *cluster, accx_scan_summary *summary, void *stream) {
  if (!g || !q) return ACCX_ERR_INVALID_ARG;
  if (!g->cnt_valid) return ACCX_ERR_NOT_READY;
  cudaStream_t s = (cudaStream_t)stream;
  ACCX_CUDA_TRY(cudaSetDevice(g->device));
  int rc = ensure_query_arrays(g, q);
  if (rc) return rc;
  const uint32_t n = g->n, m = (uint32_t)g->m;
  const accx_simq sq = accx_simq_make(eps);
  const int sms = accx_sm_count(g->device);
  ACCX_CUDA_TRY(cudaMemsetAsync(q->d_qcounters, 0, sizeof(unsigned long long) * Q_NUM, s));
  if (m && !g->key_valid.load(std::memory_order_acquire)) {
    // once per count; several threads may query one const handle, so the key
    // array is built under a lock
    static std::mutex mu_key;
    std::lock_guard<std::mutex> lk(mu_key);
    if (!g->key_valid.load(std::memory_order_relaxed)) {
      accx_graph *gm = const_cast<accx_graph *>(g);
      if (!gm->d_simkey || !gm->d_src) {
        if (!gm->d_simkey) ACCX_CUDA_TRY(accx_graph_alloc(gm, (void **)&gm->d_simkey, sizeof(float) * (size_t)m, g->home));
        if (!gm->d_src) ACCX_CUDA_TRY(accx_graph_alloc(gm, (void **)&gm->d_src, sizeof(uint32_t) * (size_t)m, g->home));
        ACCX_CUDA_TRY(accx_dev_wait(g->home));
      }
      k_simkey<<<sms * 8, 256, 0, s>>>(g->d_off, g->d_tilerow, g->d_dst, g->d_cnt, m, g->cnt_bias, gm->d_simkey,
                                       gm->d_src);
      ACCX_CUDA_TRY(cudaStreamSynchronize(s));
      gm->key_valid.store(true, std::memory_order_release);
    }
  }
  // threshold band on the keys: exact outside, simpred.h inside
  const float klo = sq.mode == 0 ? (float)sq.m2_lo * (1.0f - 4e-7f) : 0.f;
  const float khi = sq.mode == 0 ? (float)sq.m2_hi * (1.0f + 4e-7f) : 0.f;
  // the caller's similarity bytes come from the same pass: into device memory that allows
  // 8-byte stores, or into a buffer that is then copied to the host
  const bool sim_dev = sim && m && accx_is_device_ptr(sim);
  stream_block sim_tmp(s);
  uint8_t *sim_out = sim_dev && !((uintptr_t)sim & 7) ? sim : nullptr;
  if (sim && m && !sim_dev) {
    ACCX_CUDA_TRY(accx_graph_alloc(const_cast<accx_graph *>(g), &sim_tmp.p, m, s));
    sim_out = static_cast<uint8_t *>(sim_tmp.p);
  }
  if (m) k_sim_keys<<<sms * 8, 256, 0, s>>>(g->d_simkey, g->d_off, g->d_src, g->d_dst, g->d_cnt, m, g->cnt_bias, sq, klo,
                                            khi, reinterpret_cast<uint8_t *>(q->d_simbits), sim_out, q->d_qcounters);
  if (n) {
    k_cores<<<sms * 8, 256, 0, s>>>(g->d_off, n, mu, q->d_simbits, q->d_label, q->d_parent, q->d_hubmin, q->d_hubmax,
                                    q->d_corebits, q->d_big, q->d_corelist, q->d_push, q->d_qcounters);
    if (m > BIG_ROW)
      k_cores_big<<<sms * 2, 256, 0, s>>>(g->d_off, mu, q->d_simbits, q->d_big, q->d_label, q->d_corebits, q->d_push,
                                          q->d_qcounters);
  }
  if (m) {
    const auto hook = [&](auto k) {
      k<<<sms * 8, HOOK_WARPS * 32, 0, s>>>(g->d_src, g->d_dst, m, q->d_simbits, q->d_corebits, q->d_qcounters, q->d_parent);
    };
    if (m >= HOOK_OWN) hook(k_hook_words);
    hook(k_hook_lanes<true>);
    hook(k_hook_lanes<false>);
  }
  if (n) k_compress<<<sms * 4, 256, 0, s>>>(n, q->d_corebits, q->d_parent);
  if (n) k_hub_push<<<sms * 8, 256, 0, s>>>(g->d_off, g->d_dst, q->d_corelist, q->d_push, q->d_qcounters, q->d_corebits,
                                            q->d_parent, q->d_hubmin, q->d_hubmax);
  bool cl_dev = cluster && accx_is_device_ptr(cluster);
  // host clusters: through the hub minima's array, which nothing reads after this
  int32_t *cl_target = cl_dev ? cluster : cluster ? q->d_hubmin : nullptr;
  if (n) k_finish<<<sms * 4, 256, 0, s>>>(n, q->d_label, q->d_parent, q->d_hubmin, q->d_hubmax, cl_target, q->d_qcounters);
  ACCX_CUDA_TRY(cudaGetLastError());
  q->query_valid = true;
  q->pairs_valid = false;
  q->last_eps = eps;
  q->last_mu = mu;
  if (sim_dev && !sim_out) {
    k_bits_to_bytes<<<sms * 8, 256, 0, s>>>(q->d_simbits, m, sim);
    ACCX_CUDA_TRY(cudaGetLastError());
  }
  if (sim_tmp.p) {
    cudaError_t e1 = cudaMemcpyAsync(sim, sim_out, m, cudaMemcpyDeviceToHost, s);
    cudaError_t e2 = cudaStreamSynchronize(s);
    if (e1 != cudaSuccess || e2 != cudaSuccess) return ACCX_ERR_CUDA;
  }
  if (label) {
    rc = accx_copy_out(label, q->d_label, sizeof(int32_t) * n, s);
    if (rc) return rc;
  }
  if (cluster && !cl_dev && n) {
    rc = accx_copy_out(cluster, q->d_hubmin, sizeof(int32_t) * n, s);
    if (rc) return rc;
  }
  unsigned long long h[Q_NUM];
  ACCX_CUDA_TRY(cudaMemcpyAsync(h, q->d_qcounters, sizeof(h), cudaMemcpyDeviceToHost, s));
  ACCX_CUDA_TRY(cudaStreamSynchronize(s));
  q->summary.cores = (uint32_t)h[Q_CORES];
  q->summary.clusters = (uint32_t)h[Q_CLUSTERS];
  q->summary.hubs = (uint32_t)h[Q_HUBS];
  q->summary.outliers = (uint32_t)h[Q_OUTLIERS];
  q->summary.similar_entries = h[Q_SIMILAR];
  q->summary.digest = h[Q_DIGEST];
  q->summary.noncore_pairs = 0;
  if (summary) *summary = q->summary;
  return ACCX_OK;
}

extern "C" int accx_scan_query(accx_graph *g, double eps, int mu, uint8_t *sim, int32_t *label, int32_t *cluster,
                               accx_scan_summary *summary, void *stream) {
  if (!g) return ACCX_ERR_INVALID_ARG;
  return accx_scan_query_ctx(g, &g->qc, eps, mu, sim, label, cluster, summary, stream);
}

extern "C" int accx_query_ctx_create(const accx_graph *g, accx_query_ctx **out) {
  if (!g || !out) return ACCX_ERR_INVALID_ARG;
  accx_query_ctx *q = new (std::nothrow) accx_query_ctx();
  if (!q) return ACCX_ERR_OOM;
  int rc = ensure_query_arrays(g, q);
  if (rc) {
    accx_query_ctx_release(q);
    delete q;
    return rc;
  }
  *out = q;
  return ACCX_OK;
}

extern "C" int accx_query_ctx_free(accx_query_ctx *q) {
  if (!q) return ACCX_ERR_INVALID_ARG;
  accx_query_ctx_release(q);
  delete q;
  return ACCX_OK;
}

static int build_pairs(accx_graph *g, accx_query_ctx *q, cudaStream_t s) {
  if (q->pairs_valid) return ACCX_OK;
  const uint32_t n = g->n, m = (uint32_t)g->m;
  const uint32_t tiles = (m + 255) / 256;
  unsigned long long h = 0;
  ACCX_CUDA_TRY(cudaMemsetAsync(q->d_qcounters + Q_PAIRS, 0, sizeof(unsigned long long), s));
  if (m) k_pairs<256><<<tiles, 256, 0, s>>>(g->d_off, g->d_tilerow, g->d_dst, n, m, q->d_simbits, q->d_label, q->d_parent, nullptr,
                                            0, q->d_qcounters);
  ACCX_CUDA_TRY(cudaMemcpyAsync(&h, q->d_qcounters + Q_PAIRS, sizeof(h), cudaMemcpyDeviceToHost, s));
  ACCX_CUDA_TRY(cudaStreamSynchronize(s));
  if (h > q->pairs_cap) {
    accx_dev_free(q->d_pairs, nullptr);
    accx_dev_free(q->d_pairs_tmp, nullptr);
    q->d_pairs = q->d_pairs_tmp = nullptr;
    q->pairs_cap = 0;
    ACCX_CUDA_TRY(accx_graph_alloc(g, (void **)&q->d_pairs, sizeof(unsigned long long) * h, nullptr));
    ACCX_CUDA_TRY(accx_graph_alloc(g, (void **)&q->d_pairs_tmp, sizeof(unsigned long long) * h, nullptr));
    ACCX_CUDA_TRY(accx_dev_wait(nullptr));
    q->pairs_cap = h;
  }
  q->npairs = 0;
  if (h) {
    ACCX_CUDA_TRY(cudaMemsetAsync(q->d_qcounters + Q_PAIRS, 0, sizeof(unsigned long long), s));
    k_pairs<256><<<tiles, 256, 0, s>>>(g->d_off, g->d_tilerow, g->d_dst, n, m, q->d_simbits, q->d_label, q->d_parent, q->d_pairs,
                                       q->pairs_cap, q->d_qcounters);
    cub::DoubleBuffer<unsigned long long> db(q->d_pairs, q->d_pairs_tmp);
    size_t tb = 0, tb2 = 0;
    unsigned long long *d_nsel = nullptr;
    ACCX_CUDA_TRY(cub::DeviceRadixSort::SortKeys(nullptr, tb, db, (int64_t)h, 0, 64, s));
    ACCX_CUDA_TRY(cub::DeviceSelect::Unique(nullptr, tb2, q->d_pairs, q->d_pairs_tmp, d_nsel, (int64_t)h, s));
    void *tmp = nullptr;
    ACCX_CUDA_TRY(accx_graph_alloc(g, &tmp, std::max(tb, tb2) + 64, s));
    d_nsel = reinterpret_cast<unsigned long long *>(static_cast<char *>(tmp) + ((std::max(tb, tb2) + 15) & ~size_t(15)));
    cudaError_t e1 = cub::DeviceRadixSort::SortKeys(tmp, tb, db, (int64_t)h, 0, 64, s);
    unsigned long long *sorted = db.Current(), *other = db.Alternate();
    cudaError_t e2 = cub::DeviceSelect::Unique(tmp, tb2, sorted, other, d_nsel, (int64_t)h, s);
    unsigned long long nu = 0;
    cudaError_t e3 = cudaMemcpyAsync(&nu, d_nsel, sizeof(nu), cudaMemcpyDeviceToHost, s);
    cudaError_t e4 = cudaStreamSynchronize(s);
    cudaFreeAsync(tmp, s);
    if (e1 || e2 || e3 || e4) return ACCX_ERR_CUDA;
    if (other != q->d_pairs) std::swap(q->d_pairs, q->d_pairs_tmp);  // unique result lives in d_pairs
    q->npairs = nu;
  }
  q->summary.noncore_pairs = q->npairs;
  q->pairs_valid = true;
  return ACCX_OK;
}

__global__ void k_keys_to_pairs(const unsigned long long *__restrict__ keys, uint64_t np, int32_t *__restrict__ out) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < np; i += (uint64_t)gridDim.x * blockDim.x) {
    out[2 * i] = (int32_t)(keys[i] >> 32);
    out[2 * i + 1] = (int32_t)(keys[i] & 0xffffffffull);
  }
}

extern "C" int accx_scan_pairs(accx_graph *g, int32_t *pairs, uint64_t cap, uint64_t *npairs, void *stream) {
  if (!g || !npairs) return ACCX_ERR_INVALID_ARG;
  if (!g->qc.query_valid) return ACCX_ERR_NOT_READY;
  cudaStream_t s = (cudaStream_t)stream;
  ACCX_CUDA_TRY(cudaSetDevice(g->device));
  accx_query_ctx *q = &g->qc;
  int rc = build_pairs(g, q, s);
  if (rc) return rc;
  *npairs = q->npairs;
  if (!pairs) return ACCX_OK;
  if (cap < q->npairs) return ACCX_ERR_TOO_LARGE;
  if (!q->npairs) return ACCX_OK;
  stream_block block(s);
  const bool dev = accx_is_device_ptr(pairs);
  if (!dev) ACCX_CUDA_TRY(accx_graph_alloc(g, &block.p, sizeof(int32_t) * 2 * q->npairs, s));
  int32_t *tmp = dev ? pairs : static_cast<int32_t *>(block.p);
  k_keys_to_pairs<<<accx_sm_count(g->device) * 8, 256, 0, s>>>(q->d_pairs, q->npairs, tmp);
  ACCX_CUDA_TRY(cudaGetLastError());
  if (!dev) {
    cudaError_t e1 = cudaMemcpyAsync(pairs, tmp, sizeof(int32_t) * 2 * q->npairs, cudaMemcpyDeviceToHost, s);
    cudaError_t e2 = cudaStreamSynchronize(s);
    if (e1 || e2) return ACCX_ERR_CUDA;
  }
  return ACCX_OK;
}

extern "C" int accx_eps_string(double eps, char *out, size_t cap) {
  if (!out || cap == 0) return ACCX_ERR_INVALID_ARG;
  std::string s = std::to_string(eps);
  s.erase(s.find_last_not_of("0u") + 1);
  if (s.size() + 1 > cap) return ACCX_ERR_TOO_LARGE;
  memcpy(out, s.c_str(), s.size() + 1);
  return ACCX_OK;
}

// Decimal writer for the result file (the reference streams ints through an ofstream).
static inline char *put_int(char *p, int32_t v) {
  char tmp[12];
  int k = 0;
  uint32_t x = v < 0 ? (uint32_t)(-(int64_t)v) : (uint32_t)v;
  do { tmp[k++] = (char)('0' + x % 10); x /= 10; } while (x);
  if (v < 0) *p++ = '-';
  while (k) *p++ = tmp[--k];
  return p;
}

extern "C" int accx_write_result(accx_graph *g, const char *dir, double eps, int mu, void *stream) {
  if (!g || !dir) return ACCX_ERR_INVALID_ARG;
  accx_query_ctx *q = &g->qc;
  if (!q->query_valid) return ACCX_ERR_NOT_READY;
  cudaStream_t s = (cudaStream_t)stream;
  uint64_t np = 0;
  int rc = accx_scan_pairs(g, nullptr, 0, &np, stream);
  if (rc) return rc;
  std::vector<int32_t> pairs(2 * np + 2), lab(g->n + 1), par(g->n + 1);
  rc = accx_scan_pairs(g, pairs.data(), np, &np, stream);
  if (!rc) rc = accx_copy_out(lab.data(), q->d_label, sizeof(int32_t) * g->n, s);
  if (!rc) rc = accx_copy_out(par.data(), q->d_parent, sizeof(int32_t) * g->n, s);
  if (rc) return rc;
  char eps_s[512];
  rc = accx_eps_string(eps, eps_s, sizeof(eps_s));
  if (rc) return rc;
  std::string path = std::string(dir) + "/scanxp-result-" + eps_s + "-" + std::to_string(mu) + ".txt";
  FILE *f = fopen(path.c_str(), "wb");
  if (!f) return ACCX_ERR_IO;
  std::vector<char> buf(1 << 22);
  char *p = buf.data(), *lim = buf.data() + buf.size() - 64;
  bool ok = true;
  auto flush = [&]() {
    size_t len = (size_t)(p - buf.data());
    if (len && fwrite(buf.data(), 1, len, f) != len) ok = false;
    p = buf.data();
  };
  const char *hdr = "c/n vertex_id cluster_id\n";
  memcpy(p, hdr, strlen(hdr));
  p += strlen(hdr);
  for (uint32_t i = 0; i < g->n; i++) {
    if (lab[i] != ACCX_CORE) continue;
    *p++ = 'c'; *p++ = ' ';
    p = put_int(p, (int32_t)i);
    *p++ = ' ';
    p = put_int(p, par[i]);
    *p++ = '\n';
    if (p >= lim) flush();
  }
  for (uint64_t k = 0; k < np; k++) {
    *p++ = 'n'; *p++ = ' ';
    p = put_int(p, pairs[2 * k + 1]);
    *p++ = ' ';
    p = put_int(p, pairs[2 * k]);
    *p++ = '\n';
    if (p >= lim) flush();
  }
  flush();
  if (fclose(f) != 0) ok = false;
  return ok ? ACCX_OK : ACCX_ERR_IO;
}

extern "C" int accx_similar_exact(uint32_t cnn, uint32_t du, uint32_t dv, double eps) {
  accx_simq q = accx_simq_make(eps);
  return accx_similar(q, cnn, du, dv) ? 1 : 0;
}

extern "C" int accx_similar_exact_batch(uint64_t k, const uint32_t *cnn, const uint32_t *du, const uint32_t *dv,
                                        double eps, uint8_t *out) {
  if (k && (!cnn || !du || !dv || !out)) return ACCX_ERR_INVALID_ARG;
  accx_simq q = accx_simq_make(eps);
  for (uint64_t i = 0; i < k; i++) out[i] = accx_similar(q, cnn[i], du[i], dv[i]) ? 1 : 0;
  return ACCX_OK;
}

__global__ void k_cnt_digest(const int32_t *__restrict__ cnt, uint32_t m, unsigned long long *__restrict__ out) {
  unsigned long long sum = 0, dig = 0;
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < m; e = accx_entry_step(e, stride, m)) {
    const uint32_t c = (uint32_t)cnt[e];
    sum += c;
    dig += accx_mix64_dev(((unsigned long long)e << 32) | c);
  }
  for (int d = 16; d >= 1; d >>= 1) {
    sum += __shfl_xor_sync(ACCX_FULL_MASK, sum, d);
    dig += __shfl_xor_sync(ACCX_FULL_MASK, dig, d);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&out[0], sum);
    atomicAdd(&out[1], dig);
  }
}

extern "C" int accx_cn_digest(const accx_graph *g, uint64_t *sum, uint64_t *digest, void *stream) {
  if (!g) return ACCX_ERR_INVALID_ARG;
  if (!g->cnt_valid) return ACCX_ERR_NOT_READY;
  cudaStream_t s = (cudaStream_t)stream;
  unsigned long long *d = nullptr, h[2] = {0, 0};
  ACCX_CUDA_TRY(accx_dev_alloc((void **)&d, sizeof(h), s));
  cudaError_t e = cudaMemsetAsync(d, 0, sizeof(h), s);
  if (e == cudaSuccess && g->m) {
    k_cnt_digest<<<accx_sm_count(g->device) * 4, 256, 0, s>>>(g->d_cnt, (uint32_t)g->m, d);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(h, d, sizeof(h), cudaMemcpyDeviceToHost, s);
  accx_dev_free(d, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) {
    accx_set_cuda_error(e, "cn_digest", __FILE__, __LINE__);
    return ACCX_ERR_CUDA;
  }
  if (sum) *sum = h[0];
  if (digest) *digest = h[1];
  return ACCX_OK;
}
