// Degree-descending relabel of a resident graph, on the GPU.
//
// The reference offers the same preprocessing on the CPU (ReorderDegDescending +
// Reorder, scan-query/scan_xp.cpp:1145-1222, :1279-1301): vertices are renumbered
// by decreasing degree and every neighbour list is re-sorted.  Here it serves the
// counting kernels: after the relabel most probed ids (edge endpoints are mostly
// high-degree vertices) are small, so a dense shared-memory bitmap over the
// lowest ids answers most membership tests.  Counts are computed on the relabeled
// CSR and gathered back to the caller's entry order through map[e], so the
// handle's public arrays never change.
#include <cub/cub.cuh>

#include "accx_internal.h"
#include "devutil.cuh"
#include "entries.h"

// Sort keys of the vertex order: the top of the key range less the degree, so that an
// ascending stable sort of the ids by key gives degree descending, then id.  The keys have
// the bits of the entry count: fewer radix passes than a 64-bit (degree, id) key.
__global__ void k_vertex_keys(const uint32_t *__restrict__ off, uint32_t n, uint32_t top, uint32_t *__restrict__ keys,
                              uint32_t *__restrict__ ids) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    keys[v] = top - (off[v + 1] - off[v]);
    ids[v] = v;
  }
}

__global__ void k_perm(const uint32_t *__restrict__ sorted, uint32_t n, const uint32_t *__restrict__ off,
                       uint32_t *__restrict__ oldid, uint32_t *__restrict__ newid, uint32_t *__restrict__ rdeg) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint32_t v = sorted[i];
    oldid[i] = v;
    newid[v] = i;
    rdeg[i] = off[v + 1] - off[v];
  }
}

// Rows move whole: the row of old vertex u becomes row newid[u], sorted by its
// neighbours' new ids.  Relabeled rows are in non-increasing degree order, so each degree
// class is a range of rows, sorted by a kernel of its size straight from the original
// entries: it reads the row, looks up the new ids and writes the sorted row and the map.
// bounds[i] = the first row of degree <= RELABEL_CLASS[i], bounds[RELABEL_NCLASS + i] its
// first entry.
#define RELABEL_NCLASS 8
__constant__ uint32_t RELABEL_CLASS[RELABEL_NCLASS] = {4096u, 1024u, 512u, 256u, 128u, 64u, 32u, 1u};

__global__ void k_class_bounds(const uint32_t *__restrict__ rdeg, uint32_t n, const uint32_t *__restrict__ roff,
                               uint32_t *__restrict__ bounds) {
  const int i = threadIdx.x;
  if (i >= RELABEL_NCLASS) return;
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    const uint32_t mid = lo + (hi - lo) / 2;
    if (rdeg[mid] <= RELABEL_CLASS[i]) hi = mid;
    else lo = mid + 1;
  }
  bounds[i] = lo;
  bounds[RELABEL_NCLASS + i] = roff[lo];
}

// The original and the relabeled graph, as the row kernels take them.
struct relabel_view {
  const uint32_t *off;    // original offsets
  const int32_t *dst;     // original neighbours
  const uint32_t *oldid, *newid, *roff;
  uint32_t n;
  int32_t *rdst;
  uint32_t *map;
};
__device__ __forceinline__ uint32_t relabel_key(const relabel_view &g, uint32_t e) {
  const uint32_t v = (uint32_t)__ldg(g.dst + e);
  return v < g.n ? __ldg(g.newid + v) : 0xffffffffu;
}

// Rows above 4096 entries: keys and original entries for the segmented sort.  A CTA takes
// 4096 positions, which belong to one row or two (a CTA a row took 13 ms of
// a star of 16M leaves).
#define BIG_CHUNK 4096u
__global__ void __launch_bounds__(256) k_big_rows(relabel_view g, uint32_t rows, uint32_t total,
                                                  uint32_t *__restrict__ key, uint32_t *__restrict__ val) {
  const int lane = threadIdx.x & 31;
  const uint32_t chunks = total / BIG_CHUNK + (total % BIG_CHUNK ? 1u : 0u);
  for (uint32_t c = blockIdx.x; c < chunks; c += gridDim.x) {
    const uint32_t p0 = c * BIG_CHUNK;
    // the row of p0, by every warp
    uint32_t r = 0, hi = rows;
    while (hi - r > 1) {
      const uint32_t step = (hi - r + 31) / 32, q = r + (uint32_t)lane * step;
      const unsigned in = __ballot_sync(ACCX_FULL_MASK, q < hi && __ldg(g.roff + q) <= p0);
      r += (31 - __clz(in)) * step;
      hi = min(hi, r + step);
    }
    const uint32_t end = __ldg(g.roff + r + 1);
    // an entry's place in the original less its position
    const uint32_t d0 = __ldg(g.off + __ldg(g.oldid + r)) - __ldg(g.roff + r);
    const uint32_t d1 = r + 1 < rows ? __ldg(g.off + __ldg(g.oldid + r + 1)) - end : 0u;
    const uint32_t len = min(total - p0, BIG_CHUNK);
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < len; i += 256) {
      const uint32_t p = p0 + i, e = p + (p < end ? d0 : d1);
      key[p] = relabel_key(g, e);
      val[p] = e;
    }
  }
}
__global__ void k_put_big(const uint32_t *__restrict__ key, const uint32_t *__restrict__ val, uint32_t m,
                          int32_t *__restrict__ rdst, uint32_t *__restrict__ map) {
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < m; p = accx_entry_step(p, stride, m)) {
    rdst[p] = (int32_t)key[p];
    map[val[p]] = p;
  }
}

// One CTA per row of at most NT*IPT entries (rows r0..r1, CTAs loop over them):
// block radix sort over the low `bits` bits of (key, place in the row).  Padding keys are
// all ones and `bits` leaves them above every id, so they sort last.  The input
// arrangement does not matter to the sort, so loads are striped (coalesced).
template <int NT, int IPT>
__global__ void __launch_bounds__(NT) k_row_sort(relabel_view g, uint32_t r0, uint32_t r1, int bits) {
  using Sort = cub::BlockRadixSort<uint32_t, NT, IPT, uint32_t, 5>;  // 5-bit digits: 4 and 6 measured slower
  __shared__ typename Sort::TempStorage tmp;
  for (uint32_t r = r0 + blockIdx.x; r < r1; r += gridDim.x) {
    const uint32_t b = g.roff[r], d = g.roff[r + 1] - b, e0 = g.off[g.oldid[r]];
    uint32_t k[IPT], v[IPT];
#pragma unroll
    for (int i = 0; i < IPT; i++) {
      const uint32_t idx = (uint32_t)i * NT + threadIdx.x;
      k[i] = idx < d ? relabel_key(g, e0 + idx) : 0xffffffffu;
      v[i] = idx;
    }
    Sort(tmp).SortBlockedToStriped(k, v, 0, bits);
#pragma unroll
    for (int i = 0; i < IPT; i++) {
      const uint32_t idx = (uint32_t)i * NT + threadIdx.x;
      if (idx < d) {
        g.rdst[b + idx] = (int32_t)k[i];
        g.map[e0 + v[i]] = b + idx;
      }
    }
    __syncthreads();  // tmp is reused by the next row
  }
}

// One warp per row of at most 32 E entries: a bitonic network over lanes and registers
// (element 32 k + lane in register k, so loads and stores are coalesced).  One word an
// element when key and place in the row (its low log2(32 E) bits) fit (PACKED), else a
// pair.  Rows of 33 to 256 entries took a 64-thread radix sort of 256 pairs before,
// whatever their length, after a pass that wrote the pairs to memory (757 and 433 us at
// R-MAT 21; without that pass and with these sorts the whole host job takes 1.07 ms
// less).  Rows of 513 to 1024 in 32 registers a lane measured slower than the CTA radix
// sort (354 us against 268 for 257 to 1024).
__host__ __device__ constexpr int relabel_place_bits(int e) { return e == 1 ? 5 : 1 + relabel_place_bits(e / 2); }
template <int E, bool PACKED>
__global__ void __launch_bounds__(256) k_warp_row_sort(relabel_view g, uint32_t r0, uint32_t r1) {
  constexpr int SHIFT = relabel_place_bits(E);
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t r = r0 + w; r < r1; r += nw) {
    const uint32_t b = g.roff[r], d = g.roff[r + 1] - b, e0 = g.off[g.oldid[r]];
    uint32_t k[E], v[E];
#pragma unroll
    for (int i = 0; i < E; i++) {
      const uint32_t idx = 32u * i + lane, x = idx < d ? relabel_key(g, e0 + idx) : 0xffffffffu;
      k[i] = PACKED ? (idx < d ? (x << SHIFT) | idx : 0xffffffffu) : x;
      v[i] = idx;
    }
#pragma unroll
    for (uint32_t sz = 2; sz <= 32u * E; sz <<= 1) {
#pragma unroll
      for (uint32_t j = sz >> 1; j > 0; j >>= 1) {
        if (j >= 32u) {  // both elements in this lane
#pragma unroll
          for (int i = 0; i < E; i++) {
            const int o = i ^ (int)(j >> 5);
            if (o <= i) continue;
            const bool up = ((32u * i) & sz) == 0;  // ascending runs of sz alternate with descending ones
            if (up ? k[i] > k[o] : k[i] < k[o]) {
              const uint32_t t = k[i], q = v[i];
              k[i] = k[o];
              k[o] = t;
              v[i] = v[o];
              v[o] = q;
            }
          }
        } else {
#pragma unroll
          for (int i = 0; i < E; i++) {
            const uint32_t ok = __shfl_xor_sync(ACCX_FULL_MASK, k[i], j);
            // the lower lane of a pair keeps the smaller key in an ascending run
            const bool keep_min = ((lane & j) == 0) == (((32u * i + lane) & sz) == 0);
            if (PACKED) {
              k[i] = keep_min ? min(k[i], ok) : max(k[i], ok);
            } else {
              const uint32_t ov = __shfl_xor_sync(ACCX_FULL_MASK, v[i], j);
              if (keep_min ? ok < k[i] : ok > k[i]) {
                k[i] = ok;
                v[i] = ov;
              }
            }
          }
        }
      }
    }
#pragma unroll
    for (int i = 0; i < E; i++) {
      const uint32_t idx = 32u * i + lane;
      if (idx < d) {
        g.rdst[b + idx] = (int32_t)(PACKED ? k[i] >> SHIFT : k[i]);
        g.map[e0 + (PACKED ? k[i] & ((1u << SHIFT) - 1u) : v[i])] = b + idx;
      }
    }
  }
}

// Rows of at most one entry: entries p0.. of rows r0..r1 in order.
__global__ void k_put_single(relabel_view g, uint32_t r0, uint32_t r1) {
  for (uint32_t r = r0 + blockIdx.x * blockDim.x + threadIdx.x; r < r1; r += gridDim.x * blockDim.x) {
    const uint32_t b = g.roff[r];
    if (g.roff[r + 1] == b) continue;
    const uint32_t e = g.off[g.oldid[r]];
    g.rdst[b] = (int32_t)relabel_key(g, e);
    g.map[e] = b;
  }
}

// Four entries per thread and step, their index loads and then their gathers
// issued together: the gathers are random reads, bound by latency at one a thread.
// out (optional): the caller's output -- device memory, or pinned host memory mapped
// into the device's address space -- written in the same pass (each warp store is 128
// contiguous bytes, over the host link for host memory), which spares a separate copy
// of the counts (R-MAT 24: 0.63 ms to device memory).
__global__ void k_gather_counts(const int32_t *__restrict__ cnt_r, const uint32_t *__restrict__ map, uint32_t m,
                                int32_t *cnt, int32_t *out) {
  const uint32_t stride = gridDim.x * blockDim.x;
  uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
  for (; e < m && m - e > 3 * stride; e = accx_entry_step(e, 4 * stride, m)) {
    const uint32_t a = __ldg(map + e), b = __ldg(map + e + stride), c = __ldg(map + e + 2 * stride),
                   d = __ldg(map + e + 3 * stride);
    const int32_t x = __ldg(cnt_r + a), y = __ldg(cnt_r + b), z = __ldg(cnt_r + c), w = __ldg(cnt_r + d);
    cnt[e] = x;
    cnt[e + stride] = y;
    cnt[e + 2 * stride] = z;
    cnt[e + 3 * stride] = w;
    if (out) {
      out[e] = x;
      out[e + stride] = y;
      out[e + 2 * stride] = z;
      out[e + 3 * stride] = w;
    }
  }
  for (; e < m; e = accx_entry_step(e, stride, m)) {
    const int32_t x = __ldg(cnt_r + __ldg(map + e));
    cnt[e] = x;
    if (out) out[e] = x;
  }
}

// Dense rows of oriented counts (k_dense_pairs): which rows and how many hub ids.
// For every block of 1024 rows and K in 1024, 2048, 4096: the gain, in probes, of
// counting the block's prefix edges with K-bit rows.  An edge (c, b) of row c spares
// about |P(c) ∩ [0, K)| probes (its partner's ids below K; within 20 % of the true
// mean from scale 15 to 24) and costs two reads of a K-bit row, DENSE_COST probes
// each.  Beside it the same with the partner's ids below K of one edge of each row, taken by a
// hash: on a graph whose hubs are not joined to each other the first promises probes that
// nothing makes (3000 x 3000 vertices, all joined to all, 297 us, with dense rows 787, now
// 241; choosing K and M by the second alone cost R-MAT 24 3 %, the costs are fitted to the
// first).  Out: both gains, then the longest prefix of each block.
#define DENSE_COST make_float3(14.f, 22.f, 41.f)
#define DENSE_KINDS 3
#define DENSE_BLOCKS 256
#define DENSE_ROWS_MAX 192u  // blocks of 1024 ids in the default bitmap window
__global__ void __launch_bounds__(1024) k_dense_plan(const uint32_t *__restrict__ roff, const int32_t *__restrict__ rdst,
                                                     uint32_t n, float3 cost, float *__restrict__ out) {
  __shared__ float s_g[2 * DENSE_KINDS][32];
  __shared__ uint32_t s_p[32];
  const uint32_t x = blockIdx.x * 1024u + threadIdx.x;
  uint32_t p = 0;
  float gain[2 * DENSE_KINDS] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (x < n) {
    const uint32_t b = roff[x], e = roff[x + 1];
    p = accx_lower_bound(rdst, b, e, (int32_t)x) - b;
    const float c[DENSE_KINDS] = {cost.x, cost.y, cost.z};
    uint32_t hi = b + p;
#pragma unroll
    for (int k = DENSE_KINDS - 1; k >= 0; k--) {
      hi = accx_lower_bound(rdst, b, hi, (int32_t)(1024u << k));
      gain[k] = (float)p * ((float)(hi - b) - 2.f * c[k]);
    }
    if (p && blockIdx.x < DENSE_ROWS_MAX) {
      const uint32_t at = __umulhi(x * 0x9E3779B1u, p);  // the edge's place in P(x)
      const uint32_t y = (uint32_t)rdst[b + at], yb = roff[y], ye = roff[y + 1];
      // the ids below K of P(y), or of P(x) below y where y owns the edge
      uint32_t low = accx_lower_bound(rdst, yb, ye, (int32_t)min(y, 4096u));
      const uint32_t py = (y > 4096u ? accx_lower_bound(rdst, low, ye, (int32_t)y) : low) - yb;
      const bool own = p > py;
      const uint32_t lb = own ? yb : b;
      uint32_t le = own ? low : b + at;
#pragma unroll
      for (int k = DENSE_KINDS - 1; k >= 0; k--) {
        le = accx_lower_bound(rdst, lb, le, (int32_t)(1024u << k));
        gain[DENSE_KINDS + k] = (float)p * ((float)(le - lb) - 2.f * c[k]);
      }
    }
  }
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1)
#pragma unroll
    for (int k = 0; k < 2 * DENSE_KINDS; k++) gain[k] += __shfl_xor_sync(ACCX_FULL_MASK, gain[k], d);
  p = __reduce_max_sync(ACCX_FULL_MASK, p);
  if ((threadIdx.x & 31) == 0) {
    for (int k = 0; k < 2 * DENSE_KINDS; k++) s_g[k][threadIdx.x >> 5] = gain[k];
    s_p[threadIdx.x >> 5] = p;
  }
  __syncthreads();
  if (threadIdx.x < 2 * DENSE_KINDS) {
    float t = 0.f;
    for (int w = 0; w < 32; w++) t += s_g[threadIdx.x][w];
    out[threadIdx.x * DENSE_BLOCKS + blockIdx.x] = t;
  } else if (threadIdx.x == 2 * DENSE_KINDS) {
    uint32_t t = 0;
    for (int w = 0; w < 32; w++) t = max(t, s_p[w]);
    reinterpret_cast<uint32_t *>(out)[2 * DENSE_KINDS * DENSE_BLOCKS + blockIdx.x] = t;
  }
}

// Picks K and M from the gains: the rows up to the block after which no more is
// gained, at most 64 MiB of bits (half of L2), and only if that spares more than the
// two extra launches (DENSE_MIN probes) and the rows' sampled edges gain too.
#define DENSE_MIN 4e6f
static void dense_choose(accx_graph *g, const float *out) {
  const uint32_t blocks = (g->n + 1023u) / 1024u < DENSE_BLOCKS ? (g->n + 1023u) / 1024u : DENSE_BLOCKS;
  float best = DENSE_MIN;
  for (uint32_t k = 0; k < DENSE_KINDS; k++) {
    const uint32_t K = 1024u << k, lim = (64u << 20) / (K / 8u) / 1024u;
    float acc = 0.f, sampled = 0.f;
    for (uint32_t i = 0; i < blocks && i < lim && i < DENSE_ROWS_MAX; i++) {
      acc += out[k * DENSE_BLOCKS + i];
      sampled += out[(DENSE_KINDS + k) * DENSE_BLOCKS + i];
      if (acc > best && sampled > 0.f) {
        best = acc;
        g->dense_k = K;
        g->dense_m = (i + 1) * 1024u < g->n ? (i + 1) * 1024u : g->n;
      }
    }
  }
  g->plan_rows = blocks * 1024u;
  for (uint32_t i = 0; i < blocks; i++) {
    const uint32_t p = reinterpret_cast<const uint32_t *>(out)[2 * DENSE_KINDS * DENSE_BLOCKS + i];
    if (p > g->plan_maxpre) g->plan_maxpre = p;
  }
}

int accx_relabel_gather(accx_graph *g, int32_t *out, cudaStream_t s) {
  const uint32_t m = (uint32_t)g->m;
  if (!m) return ACCX_OK;
  k_gather_counts<<<accx_sm_count(g->device) * 8, 256, 0, s>>>(g->d_rcnt, g->d_rmap, m, g->d_cnt, out);
  ACCX_CUDA_TRY(cudaGetLastError());
  return ACCX_OK;
}

extern "C" int accx_graph_relabel(accx_graph *g, void *stream) {
  if (!g) return ACCX_ERR_INVALID_ARG;
  if (g->d_roff) return ACCX_OK;
  cudaStream_t s = (cudaStream_t)stream;
  ACCX_CUDA_TRY(cudaSetDevice(g->device));
  const uint32_t n = g->n, m = (uint32_t)g->m;
  const int grid = accx_sm_count(g->device) * 8;
  // temporaries: vertex keys and ids (two buffers each; the plan lies in them later),
  // degrees, class bounds
  uint32_t *vtmp = nullptr, *rdeg = nullptr, *key = nullptr;
  void *tmp = nullptr;
  size_t tb = 0;
  int rc = ACCX_OK;
  const size_t vn = ((size_t)n + 64) & ~(size_t)63;
  do {
    if (accx_graph_alloc(g, (void **)&vtmp, sizeof(uint32_t) * (4 * vn + (2 * DENSE_KINDS + 1) * DENSE_BLOCKS), g->home) != cudaSuccess ||
        accx_graph_alloc(g, (void **)&rdeg, sizeof(uint32_t) * (vn + 2 * RELABEL_NCLASS + 2), g->home) != cudaSuccess ||
        accx_graph_alloc(g, (void **)&g->d_roff, sizeof(uint32_t) * ((size_t)n + 1), g->home) != cudaSuccess ||
        accx_graph_alloc(g, (void **)&g->d_rdst, sizeof(int32_t) * ((size_t)m + ACCX_DST_PAD), g->home) != cudaSuccess ||
        accx_graph_alloc(g, (void **)&g->d_rmap, sizeof(uint32_t) * ((size_t)m + 1), g->home) != cudaSuccess ||
        accx_graph_alloc(g, (void **)&g->d_rcnt, sizeof(int32_t) * ((size_t)m + 1), g->home) != cudaSuccess ||
        accx_graph_alloc(g, (void **)&g->d_oldid, sizeof(uint32_t) * ((size_t)n + 1), g->home) != cudaSuccess ||
        accx_graph_alloc(g, (void **)&g->d_newid, sizeof(uint32_t) * ((size_t)n + 1), g->home) != cudaSuccess) {
      rc = ACCX_ERR_OOM;
      break;
    }
    uint32_t *bounds = rdeg + vn;
    // sort keys: ids need `bits` bits with the all-ones pattern left above every id, degrees `dbits`
    int bits = 1, dbits = 1;
    while (bits < 32 && (1ull << bits) <= (unsigned long long)n) bits++;
    while (dbits < 32 && (1ull << dbits) <= (unsigned long long)m) dbits++;
    cub::DoubleBuffer<uint32_t> dk(vtmp, vtmp + vn), dv(vtmp + 2 * vn, vtmp + 3 * vn);
    size_t b1 = 0, b2 = 0;
    if (cub::DeviceRadixSort::SortPairs(nullptr, b1, dk, dv, (int64_t)n, 0, dbits, s) != cudaSuccess ||
        cub::DeviceScan::ExclusiveSum(nullptr, b2, rdeg, g->d_roff, (int64_t)n + 1, s) != cudaSuccess) {
      rc = ACCX_ERR_CUDA;
      break;
    }
    tb = b1 > b2 ? b1 : b2;
    if (accx_graph_alloc(g, &tmp, tb + 16, g->home) != cudaSuccess) { rc = ACCX_ERR_OOM; break; }
    if (accx_dev_wait(g->home) != cudaSuccess) { rc = ACCX_ERR_CUDA; break; }
    // 1. vertex order: degree descending, ties by id
    if (n) {
      k_vertex_keys<<<grid, 256, 0, s>>>(g->d_off, n, (uint32_t)((1ull << dbits) - 1), vtmp, vtmp + 2 * vn);
      if (cub::DeviceRadixSort::SortPairs(tmp, tb, dk, dv, (int64_t)n, 0, dbits, s) != cudaSuccess) { rc = ACCX_ERR_CUDA; break; }
      k_perm<<<grid, 256, 0, s>>>(dv.Current(), n, g->d_off, g->d_oldid, g->d_newid, rdeg);
    }
    if (cudaMemsetAsync(rdeg + n, 0, sizeof(uint32_t), s) != cudaSuccess) { rc = ACCX_ERR_CUDA; break; }
    if (cub::DeviceScan::ExclusiveSum(tmp, tb, rdeg, g->d_roff, (int64_t)n + 1, s) != cudaSuccess) { rc = ACCX_ERR_CUDA; break; }
    if (m) {
      // 2. every row sorted by its neighbours' new ids, with a kernel sized for its degree class
      const relabel_view view{g->d_off, g->d_dst, g->d_oldid, g->d_newid, g->d_roff, n, g->d_rdst, g->d_rmap};
      uint32_t hb[2 * RELABEL_NCLASS];
      k_class_bounds<<<1, 32, 0, s>>>(rdeg, n, g->d_roff, bounds);
      if (cudaMemcpyAsync(hb, bounds, sizeof(hb), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
          cudaStreamSynchronize(s) != cudaSuccess) {
        rc = ACCX_ERR_CUDA;
        break;
      }
      const uint32_t *rb = hb, *pb = hb + RELABEL_NCLASS;  // class row bounds and their entry positions
      const int sms = accx_sm_count(g->device);
      // rows above 4096 entries: segmented radix sort (one CTA per row)
      if (rb[0] > 0) {
        size_t b3 = 0;
        uint32_t *none = nullptr;
        if (cub::DeviceSegmentedRadixSort::SortPairs(nullptr, b3, none, none, none, none, (int64_t)pb[0], (int64_t)rb[0],
                                                     g->d_roff, g->d_roff + 1, 0, bits, s) != cudaSuccess) {
          rc = ACCX_ERR_CUDA;
          break;
        }
        // keys and entries, sorted into a second pair; the scratch behind them
        const size_t kn = ((size_t)pb[0] + 64) & ~(size_t)63;
        if (accx_graph_alloc(g, (void **)&key, sizeof(uint32_t) * 4 * kn + b3 + 16, g->home) != cudaSuccess) { rc = ACCX_ERR_OOM; break; }
        if (accx_dev_wait(g->home) != cudaSuccess) { rc = ACCX_ERR_CUDA; break; }
        uint32_t *val = key + kn, *key2 = key + 2 * kn, *val2 = key + 3 * kn;
        const uint32_t chunks = pb[0] / BIG_CHUNK + 1;
        k_big_rows<<<chunks < (uint32_t)sms * 8 ? chunks : sms * 8, 256, 0, s>>>(view, rb[0], pb[0], key, val);
        if (cub::DeviceSegmentedRadixSort::SortPairs(key + 4 * kn, b3, key, key2, val, val2, (int64_t)pb[0], (int64_t)rb[0],
                                                     g->d_roff, g->d_roff + 1, 0, bits, s) != cudaSuccess) {
          rc = ACCX_ERR_CUDA;
          break;
        }
        k_put_big<<<sms * 8, 256, 0, s>>>(key2, val2, pb[0], g->d_rdst, g->d_rmap);
      }
      auto rows_grid = [&](uint32_t rows, int per_sm) { return (int)(rows < (uint32_t)(sms * per_sm) ? rows : sms * per_sm); };
      auto warps_grid = [&](uint32_t rows) { return rows_grid((rows + 7) / 8, 16); };
      // words of (key, place) where both fit
      auto fits = [&](int e) { return bits + relabel_place_bits(e) <= 32; };
      if (rb[1] > rb[0]) k_row_sort<256, 16><<<rows_grid(rb[1] - rb[0], 8), 256, 0, s>>>(view, rb[0], rb[1], bits);
      if (rb[2] > rb[1])
        k_row_sort<128, 8><<<rows_grid(rb[2] - rb[1], 16), 128, 0, s>>>(view, rb[1], rb[2], bits);
      if (rb[3] > rb[2] && fits(16))
        k_warp_row_sort<16, true><<<warps_grid(rb[3] - rb[2]), 256, 0, s>>>(view, rb[2], rb[3]);
      else if (rb[3] > rb[2])
        k_row_sort<128, 8><<<rows_grid(rb[3] - rb[2], 16), 128, 0, s>>>(view, rb[2], rb[3], bits);
      if (rb[4] > rb[3])
        (fits(8) ? k_warp_row_sort<8, true> : k_warp_row_sort<8, false>)<<<warps_grid(rb[4] - rb[3]), 256, 0, s>>>(view, rb[3], rb[4]);
      if (rb[5] > rb[4])
        (fits(4) ? k_warp_row_sort<4, true> : k_warp_row_sort<4, false>)<<<warps_grid(rb[5] - rb[4]), 256, 0, s>>>(view, rb[4], rb[5]);
      if (rb[6] > rb[5])
        (fits(2) ? k_warp_row_sort<2, true> : k_warp_row_sort<2, false>)<<<warps_grid(rb[6] - rb[5]), 256, 0, s>>>(view, rb[5], rb[6]);
      if (rb[7] > rb[6])
        (fits(1) ? k_warp_row_sort<1, true> : k_warp_row_sort<1, false>)<<<warps_grid(rb[7] - rb[6]), 256, 0, s>>>(view, rb[6], rb[7]);
      if (m > pb[7]) k_put_single<<<sms * 8, 256, 0, s>>>(view, rb[7], n);
    }
    if (cudaMemsetAsync(g->d_rdst + m, 0xff, sizeof(int32_t) * ACCX_DST_PAD, s) != cudaSuccess) { rc = ACCX_ERR_CUDA; break; }
    if ((rc = accx_tilerow_build(g, g->d_roff, &g->d_rtilerow, s)) != ACCX_OK) break;
    // 3. the dense rows of oriented counts
    float plan[(2 * DENSE_KINDS + 1) * DENSE_BLOCKS];
    const bool dense = m && n;
    if (dense) {
      const uint32_t pb = (n + 1023u) / 1024u;
      float *d_plan = reinterpret_cast<float *>(vtmp + 4 * vn);
      k_dense_plan<<<pb < DENSE_BLOCKS ? pb : DENSE_BLOCKS, 1024, 0, s>>>(g->d_roff, g->d_rdst, n, DENSE_COST, d_plan);
      if (cudaMemcpyAsync(plan, d_plan, sizeof(plan), cudaMemcpyDeviceToHost, s) != cudaSuccess) { rc = ACCX_ERR_CUDA; break; }
    }
    if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(s) != cudaSuccess) { rc = ACCX_ERR_CUDA; break; }
    if (dense) dense_choose(g, plan);
  } while (0);
  if (rc) {
    cudaGetLastError();
    cudaStreamSynchronize(s);  // nothing of this call may still be running on the temporaries
  }
  void *temps[] = {vtmp, rdeg, key, tmp};
  accx_dev_free_all(temps, 4, g->home);
  if (!rc && g->d_rev_orig) {  // counts run on the relabeled CSR from now on
    accx_dev_free(g->d_rev_orig, g->home);
    g->d_rev_orig = nullptr;
  }
  if (rc) {
    for (void **p : {(void **)&g->d_roff, (void **)&g->d_rdst, (void **)&g->d_rmap, (void **)&g->d_rcnt,
                     (void **)&g->d_oldid, (void **)&g->d_newid, (void **)&g->d_rtilerow}) {
      accx_dev_free(*p, g->home);
      *p = nullptr;
    }
  }
  return rc;
}

extern "C" int accx_graph_is_relabeled(const accx_graph *g) { return g && g->d_roff ? 1 : 0; }

extern "C" int accx_graph_relabeled_csr(const accx_graph *g, uint32_t *roff, int32_t *rdst, uint32_t *map,
                                        uint32_t *oldid, void *stream) {
  if (!g) return ACCX_ERR_INVALID_ARG;
  if (!g->d_roff) return ACCX_ERR_NOT_READY;
  cudaStream_t s = (cudaStream_t)stream;
  int rc = ACCX_OK;
  if (!rc && roff) rc = accx_copy_out(roff, g->d_roff, sizeof(uint32_t) * ((size_t)g->n + 1), s);
  if (!rc && rdst) rc = accx_copy_out(rdst, g->d_rdst, sizeof(int32_t) * (size_t)g->m, s);
  if (!rc && map) rc = accx_copy_out(map, g->d_rmap, sizeof(uint32_t) * (size_t)g->m, s);
  if (!rc && oldid) rc = accx_copy_out(oldid, g->d_oldid, sizeof(uint32_t) * (size_t)g->n, s);
  return rc;
}
