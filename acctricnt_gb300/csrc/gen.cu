// Device-side synthetic graph generators and the edge-list -> CSR builder.
//
// The builder does on the GPU what the reference's EdgeListToBinsConverter does
// on the host (scan-query/converter/EdgeListToBinsConverter.cpp:24-126): keep each
// undirected edge once, drop self loops, sort, and emit degrees plus sorted
// adjacency lists.  Unlike the converter it counts degrees after removing
// duplicates, so duplicated input edges cannot produce inconsistent files.
// Sorting and unique-selection use CUB (library code; this is input
// preparation, not the counting path).
#include <cub/cub.cuh>

#include <vector>

#include "accx_internal.h"
#include "gen_host.h"

// Entry keys: (source << b) | neighbour with b = the bits of an id, so that a sort passes
// over 2b bits instead of 64 (five of eight radix passes for a million vertices) and
// graphs of up to 65536 vertices have 32-bit keys.  All 2b bits set would be a self
// loop, so that is the key of dropped draws: they sort last.
template <typename K>
__global__ void k_gen_keys(int kind, uint64_t seed_mix, uint64_t draws, uint32_t n, int scale,
                           accx_rmat_thresholds t, const uint64_t *__restrict__ cdf, int b, K *__restrict__ keys) {
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const K none = accx_key_none<K>(b);
  for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < draws; k += stride) {
    uint32_t u, v;
    if (kind == ACCX_GEN_RMAT) accx_rmat_edge(seed_mix, k, scale, t, &u, &v);
    else if (kind == ACCX_GEN_ER) accx_er_edge(seed_mix, k, n, &u, &v);
    else accx_cl_edge(seed_mix, k, cdf, n, &u, &v);
    keys[2 * k] = u != v ? ((K)u << b) | v : none;
    keys[2 * k + 1] = u != v ? ((K)v << b) | u : none;
  }
}

// off[w] = first index whose source is >= w; dst = low bits.
template <typename K>
__global__ void k_keys_to_csr(const K *__restrict__ keys, uint64_t nk, uint32_t n, int b, uint32_t *__restrict__ off,
                              int32_t *__restrict__ dst) {
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i <= nk; i += stride) {
    int64_t u_prev = (i == 0) ? -1 : (int64_t)(keys[i - 1] >> b);
    int64_t u_cur = (i == nk) ? (int64_t)n : (int64_t)(keys[i] >> b);
    for (int64_t w = u_prev + 1; w <= u_cur; w++) off[w] = (uint32_t)i;
    if (i < nk) dst[i] = (int32_t)(keys[i] & (((K)1 << b) - 1));
  }
}

// res = the distinct keys without the dropped draws' one, and the caller's defect flag.
template <typename K>
__global__ void k_key_count(const K *__restrict__ uniq, const unsigned long long *__restrict__ nsel, int b,
                            const int *__restrict__ bad, unsigned long long *__restrict__ res) {
  const unsigned long long nu = *nsel;
  res[0] = nu && uniq[nu - 1] == accx_key_none<K>(b) ? nu - 1 : nu;
  res[1] = bad ? (unsigned long long)*bad : 0ull;
}

// Sort, unique, drop the dropped draws' key, and fill g->d_off/d_dst.  One wait for the
// number of entries and one at the end.
template <typename K>
static int build_csr(accx_graph *g, K *d_keys, uint64_t nkeys, uint32_t n, const int *d_bad, cudaStream_t s) {
  const int b = accx_key_bits(n);
  char *tmp = nullptr;
  size_t t1 = 0, t2 = 0;
  unsigned long long *d_res = nullptr;  // nsel, then k_key_count's
  int rc = ACCX_OK;
  do {
    cub::DoubleBuffer<K> db(d_keys, nullptr);
    if (cub::DeviceRadixSort::SortKeys(nullptr, t1, db, (int64_t)nkeys, 0, 2 * b, s) != cudaSuccess ||
        cub::DeviceSelect::Unique(nullptr, t2, d_keys, d_keys, d_res, (int64_t)nkeys, s) != cudaSuccess) { rc = ACCX_ERR_CUDA; break; }
    const size_t alt = (sizeof(K) * (nkeys ? nkeys : 1) + 255) & ~(size_t)255;
    size_t tb = t1 > t2 ? t1 : t2;
    if (accx_dev_alloc((void **)&tmp, alt + 256 + (tb ? tb : 1), s) != cudaSuccess) {
      // no room to sort them, but a defect of the edges comes first
      int bad = 0;
      rc = d_bad && cudaMemcpyAsync(&bad, d_bad, sizeof(bad), cudaMemcpyDeviceToHost, s) == cudaSuccess &&
           cudaStreamSynchronize(s) == cudaSuccess && bad ? ACCX_ERR_RANGE : ACCX_ERR_OOM;
      cudaGetLastError();
      break;
    }
    d_res = reinterpret_cast<unsigned long long *>(tmp + alt);
    void *d_tmp = tmp + alt + 256;
    db = cub::DoubleBuffer<K>(d_keys, reinterpret_cast<K *>(tmp));
    if (cub::DeviceRadixSort::SortKeys(d_tmp, tb, db, (int64_t)nkeys, 0, 2 * b, s) != cudaSuccess) { rc = ACCX_ERR_CUDA; break; }
    K *sorted = db.Current(), *uniq = db.Alternate();
    if (cub::DeviceSelect::Unique(d_tmp, tb, sorted, uniq, d_res, (int64_t)nkeys, s) != cudaSuccess) { rc = ACCX_ERR_CUDA; break; }
    k_key_count<<<1, 1, 0, s>>>(uniq, d_res, b, d_bad, d_res + 1);
    unsigned long long h[2] = {0, 0};
    if (cudaMemcpyAsync(h, d_res + 1, sizeof(h), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess) { rc = ACCX_ERR_CUDA; break; }
    if (h[1]) { rc = ACCX_ERR_RANGE; break; }
    const unsigned long long nu = h[0];
    if (nu >= (1ull << 32) - ACCX_DST_PAD) { rc = ACCX_ERR_TOO_LARGE; break; }
    g->n = n;
    g->m = nu;
    if (accx_dev_alloc((void **)&g->d_off, sizeof(uint32_t) * ((size_t)n + 1), g->home) != cudaSuccess ||
        accx_dev_alloc((void **)&g->d_dst, sizeof(int32_t) * ((size_t)nu + ACCX_DST_PAD), g->home) != cudaSuccess) { rc = ACCX_ERR_OOM; break; }
    if (g->home != s && accx_dev_wait(g->home) != cudaSuccess) { rc = ACCX_ERR_CUDA; break; }
    if (cudaMemsetAsync(g->d_dst + nu, 0xff, sizeof(int32_t) * ACCX_DST_PAD, s) != cudaSuccess) { rc = ACCX_ERR_CUDA; break; }
    int grid = accx_grid_for(g->device, 256, 8);
    k_keys_to_csr<<<grid, 256, 0, s>>>(uniq, nu, n, b, g->d_off, g->d_dst);
    if (cudaGetLastError() != cudaSuccess) { rc = ACCX_ERR_CUDA; break; }
    if ((rc = accx_tilerow_build(g, g->d_off, &g->d_tilerow, s)) != ACCX_OK) break;
    if (cudaStreamSynchronize(s) != cudaSuccess) { rc = ACCX_ERR_CUDA; break; }
  } while (0);
  if (rc == ACCX_ERR_CUDA || rc == ACCX_ERR_OOM) cudaGetLastError();
  accx_dev_free(tmp, s);
  return rc;
}

int accx_build_csr_from_keys(accx_graph *g, void *d_keys, uint64_t nkeys, uint32_t n, const int *d_bad,
                             cudaStream_t s) {
  return accx_key_size(n) == 4 ? build_csr(g, static_cast<uint32_t *>(d_keys), nkeys, n, d_bad, s)
                               : build_csr(g, static_cast<unsigned long long *>(d_keys), nkeys, n, d_bad, s);
}

extern "C" int accx_graph_generate(const accx_gen_params *p, void *stream, accx_graph **out) {
  if (!p || !out) return ACCX_ERR_INVALID_ARG;
  *out = nullptr;
  uint32_t n;
  uint64_t draws;
  int rc = accx_gen_shape(p, &n, &draws);
  if (rc) return rc;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    return ACCX_ERR_NO_DEVICE;
  }
  cudaStream_t s = (cudaStream_t)stream;
  accx_graph *g = new (std::nothrow) accx_graph();
  if (!g) return ACCX_ERR_OOM;
  cudaGetDevice(&g->device);
  g->home = s;
  g->symmetric = true;  // the edge stream is symmetrised
  void *d_keys = nullptr;
  uint64_t *d_cdf = nullptr;
  do {
    if (accx_dev_alloc(&d_keys, accx_key_size(n) * draws * 2, s) != cudaSuccess) { rc = ACCX_ERR_OOM; break; }
    accx_rmat_thresholds t{};
    if (p->kind == ACCX_GEN_RMAT) t = accx_rmat_make(p->q0, p->q1, p->q2);
    if (p->kind == ACCX_GEN_CHUNG_LU) {
      std::vector<uint64_t> cdf;
      accx_chung_lu_cdf(n, draws, p->q0, p->q1, cdf);
      if (accx_dev_alloc((void **)&d_cdf, sizeof(uint64_t) * cdf.size(), s) != cudaSuccess) { rc = ACCX_ERR_OOM; break; }
      if (cudaMemcpyAsync(d_cdf, cdf.data(), sizeof(uint64_t) * cdf.size(), cudaMemcpyHostToDevice, s) != cudaSuccess ||
          cudaStreamSynchronize(s) != cudaSuccess) { rc = ACCX_ERR_CUDA; break; }
    }
    int grid = accx_grid_for(g->device, 256, 8);
    const int b = accx_key_bits(n);
    if (accx_key_size(n) == 4)
      k_gen_keys<<<grid, 256, 0, s>>>(p->kind, accx_mix64(p->seed), draws, n, (int)p->p0, t, d_cdf, b,
                                      static_cast<uint32_t *>(d_keys));
    else
      k_gen_keys<<<grid, 256, 0, s>>>(p->kind, accx_mix64(p->seed), draws, n, (int)p->p0, t, d_cdf, b,
                                      static_cast<unsigned long long *>(d_keys));
    if (cudaGetLastError() != cudaSuccess) { rc = ACCX_ERR_CUDA; break; }
    if (d_cdf && (cudaStreamSynchronize(s) != cudaSuccess)) { rc = ACCX_ERR_CUDA; break; }
    rc = accx_build_csr_from_keys(g, d_keys, draws * 2, n, nullptr, s);
  } while (0);
  if (rc == ACCX_ERR_CUDA || rc == ACCX_ERR_OOM) cudaGetLastError();
  accx_dev_free(d_keys, s);
  accx_dev_free(d_cdf, s);
  if (rc) {
    accx_graph_free(g);
    return rc;
  }
  *out = g;
  return ACCX_OK;
}
