// Oriented all-edge counting: common-neighbour counts as triangle credits.
//
// |N(u) ∩ N(v)| for an edge (u,v) is the number of triangles through it.  With
// the prefix P(x) = N(x) ∩ [0, x) (the neighbours with smaller ids; after the
// degree-descending relabel the higher-degree ones, at most sqrt(2m) ids), every
// triangle a < b < c is met exactly once: on the edge (c,b), as the id a common
// to P(c) ∩ [0,b) and P(b).  Each meeting adds one to the three entries (c,b),
// (c,a) and (b,a); a final pass adds the two entries of every undirected edge
// and writes the sum (plus the bias) to both.  The per-edge kernels are those of
// the direct path with prefix lists: an owner (the endpoint with the longer
// prefix, ties: smaller id) and a partner, the probe side cut at the smaller id.
//
// Credits are fire-and-forget atomics (RED): the partner-side entry of a match
// is the entry being read, so a warp's credits land in the lines it just loaded.
// The bitmap kernel keeps the owner-side credits in shared counters (one per
// prefix entry, found as the word's base rank + a popcount) and adds them to
// HBM once per work item.
//
// Included by count.cu after the shared counting definitions.
#pragma once

// ids per lane in a full piece of a long probe list (two per 8-byte load); at R-MAT
// scale 24, 8 measured 4% slower
#define LONG_UNROLL 16

// pre[u] = |N(u) ∩ [0, u)|; vinfo (optional) = (off[u], pre[u]) packed, so that a
// kernel looking up a random partner reads one 8-byte record instead of two arrays
// (on graphs without locality, e.g. Erdos-Renyi, each lookup is a DRAM access).
__global__ void k_pre(const uint32_t *__restrict__ off, const int32_t *__restrict__ dst, uint32_t n,
                      uint32_t *__restrict__ pre, uint2 *__restrict__ vinfo) {
  for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < n; u += gridDim.x * blockDim.x) {
    const uint32_t b = __ldg(off + u), e = __ldg(off + u + 1);
    const uint32_t p = accx_lower_bound(dst, b, e, (int32_t)u) - b;
    pre[u] = p;
    if (vinfo) vinfo[u] = make_uint2(b, p);
  }
}

// Reverse entries: rev[e] = position of u in N(v) for every entry e = (u,v).
// One thread per entry e = (v,u) with u > v searches v in u's prefix (a short
// list after the degree relabel) and sets both directions; entries without a
// reverse (asymmetric input) keep the 0xffffffff the array was filled with.
template <int TILE>
__global__ void __launch_bounds__(TILE) k_rev_build(const uint32_t *__restrict__ off,
                                                    const uint32_t *__restrict__ tilerow,
                                                    const int32_t *__restrict__ dst,
                                                    const uint32_t *__restrict__ pre, uint32_t n, uint32_t m,
                                                    uint32_t *__restrict__ rev) {
  __shared__ accx_tile_rows<TILE> sh;
  const uint32_t base = blockIdx.x * (uint32_t)TILE;
  const uint32_t e = base + threadIdx.x;
  const uint32_t v = accx_tile_row<TILE>(off, tilerow, n, m, base, e, &sh);
  if (e >= m) return;
  const uint32_t u = (uint32_t)dst[e];
  if (u <= v) return;
  const uint32_t ub = __ldg(off + u), ue = ub + __ldg(pre + u);
  const uint32_t r = accx_lower_bound(dst, ub, ue, (int32_t)v);
  if (r < ue && __ldg(dst + r) == (int32_t)v) {
    rev[e] = r;
    rev[r] = e;
  }
}

// The two prefix ranges of an owned edge (x owner, y = dst[e]), each cut at
// min(x, y): ids from there up cannot be common to both prefixes.  The cut of
// P(x) at y < x is the entry e itself; the cut of P(y) at x < y is x's position
// in N(y), the reverse entry.
__device__ __forceinline__ void accx_or_ranges(const uint32_t *__restrict__ off, const uint32_t *__restrict__ pre,
                                               const uint32_t *__restrict__ rev, uint32_t x, uint32_t y, uint32_t e,
                                               uint32_t *xb, uint32_t *xe, uint32_t *yb, uint32_t *ye) {
  *xb = __ldg(off + x);
  *xe = *xb + __ldg(pre + x);
  *yb = __ldg(off + y);
  *ye = *yb + __ldg(pre + y);
  if (y < x) {
    *xe = min(*xe, e);
  } else {
    const uint32_t r = __ldg(rev + e);
    *ye = (r >= *yb && r < *ye) ? r : *yb;
  }
}

__global__ void __launch_bounds__(MERGE_WARPS * 32) k_merge_or(const uint32_t *__restrict__ off,
                                                                const int32_t *__restrict__ dst,
                                                                const uint32_t *__restrict__ pre,
                                                                const uint32_t *__restrict__ rev,
                                                                const uint2 *__restrict__ list, uint32_t list_cap,
                                                                unsigned long long *__restrict__ ctr,
                                                                int32_t *__restrict__ cnt) {
  __shared__ __align__(16) int32_t buf[MERGE_WARPS][2][MERGE_WIN];
  unsigned long long found = 0;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned long long total = ctr[C_MERGE];
  if (total > list_cap) total = list_cap;
  const unsigned long long nw = (unsigned long long)gridDim.x * MERGE_WARPS;
  for (unsigned long long it = (unsigned long long)blockIdx.x * MERGE_WARPS + w; it < total; it += nw) {
    const uint2 p = list[it];
    const uint32_t x = p.x, e = p.y, y = (uint32_t)__ldg(dst + e);
    uint32_t xb, xe, yb, ye;
    accx_or_ranges(off, pre, rev, x, y, e, &xb, &xe, &yb, &ye);
    const uint32_t c = accx_warp_merge_credit(dst, xb, xe, yb, ye, buf[w][0], buf[w][1], lane, cnt);
    if (lane == 0 && c) atomicAdd(cnt + (y < x ? e : ye), (int32_t)c);  // the edge's prefix entry
    found += c;
    __syncwarp();
  }
  if (lane == 0 && found) atomicAdd(&ctr[C_MATCH + ACCX_KIND_MERGE], found);
}

// One galloping edge by G lanes: the lanes take the partner's ids in order and
// binary-search each in the owner's prefix; every round starts at the position the
// group's last lane reached.  Credits both entries of a match; returns the matches.
template <int G>
__device__ __forceinline__ uint32_t or_gallop_group(const int32_t *__restrict__ dst, uint32_t xb, uint32_t xe,
                                                    uint32_t yb, uint32_t ye, int gl, unsigned gmask,
                                                    int32_t *__restrict__ cnt) {
  uint32_t c = 0, lo = xb;
  for (uint32_t j0 = yb; j0 < ye && lo < xe; j0 += G) {
    const uint32_t j = j0 + (uint32_t)gl;
    uint32_t pos = xe;
    if (j < ye) {
      const int32_t id = __ldg(dst + j);
      pos = accx_lower_bound(dst, lo, xe, id);
      if (pos < xe && __ldg(dst + pos) == id) {
        c++;
        atomicAdd(cnt + pos, 1);
        atomicAdd(cnt + j, 1);
      }
    }
    const uint32_t last = (ye - j0 >= (uint32_t)G) ? (uint32_t)G - 1u : (ye - j0 - 1);
    lo = __shfl_sync(gmask, pos, (int)last, G);
  }
#pragma unroll
  for (int d = G / 2; d >= 1; d >>= 1) c += __shfl_xor_sync(gmask, c, d, G);
  return c;
}

// Galloping edges.  An edge's records are its list entry, the partner range that classify
// wrote (sl[e], already cut at min(x, y)) and the owner's offset and prefix length
// (vinfo): y < x exactly when e lies in x's prefix, and then the owner's range is cut at e
// and the edge's credit goes to e; otherwise to the end of the partner range (x's
// position in N(y)).  Two kernels, each of which returns at once when the edges are the
// other's: where the partner lists average more than GALLOP_MEAN ids, groups of G lanes
// take one edge each (k_gallop_or), else a lane does (k_gallop_lane).  Groups also take fewer
// edges than k_gallop_lane has lanes (GALLOP_FEW): no lane has a second one then, and the
// longest is the time (counts, us, lanes / groups: R-MAT 14 with 111K galloping edges in its
// own numbering 196 / 97, R-MAT 13 152 / 79, a mixed table at R-MAT 12 148 / 118; cliques of
// 20 with 380K 71 / 114, Erdos-Renyi with 1M 91 / 143).
#define GALLOP_MEAN 24ull
#define GALLOP_FEW 196608ull
__device__ __forceinline__ bool or_gallop_long(const unsigned long long *__restrict__ ctr) {
  return ctr[C_WORK + ACCX_KIND_GALLOP] > GALLOP_MEAN * ctr[C_EDGES + ACCX_KIND_GALLOP] ||
         ctr[C_EDGES + ACCX_KIND_GALLOP] < GALLOP_FEW;
}
struct or_gallop_edge {
  uint32_t xb, xe, yb, ye, at;  // owner range, partner range, the edge's prefix entry
};
__device__ __forceinline__ or_gallop_edge or_gallop_get(uint2 p, uint2 r, uint2 xi) {
  const uint32_t xp = xi.x + xi.y, ye = r.x + (r.y & ~OR_SL_GALLOP);
  return or_gallop_edge{xi.x, min(xp, p.y), r.x, ye, p.y < xp ? p.y : ye};
}

template <int G>
__global__ void __launch_bounds__(MERGE_WARPS * 32, 8) k_gallop_or(const uint2 *__restrict__ vinfo,
                                                                    const int32_t *__restrict__ dst,
                                                                    const uint2 *__restrict__ sl,
                                                                    const uint2 *__restrict__ list, uint32_t list_cap,
                                                                    unsigned long long *__restrict__ ctr,
                                                                    int32_t *__restrict__ cnt) {
  static_assert(G == 8 || G == 16 || G == 32, "group size");
  if (!or_gallop_long(ctr)) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int sub = lane / G, gl = lane % G;
  const unsigned gmask = G == 32 ? ACCX_FULL_MASK : (((1u << G) - 1u) << (sub * G));
  unsigned long long found = 0;
  unsigned long long total = ctr[C_GALLOP];
  if (total > list_cap) total = list_cap;
  const unsigned long long ng = (unsigned long long)gridDim.x * MERGE_WARPS * (32 / G);
  for (unsigned long long it = ((unsigned long long)blockIdx.x * MERGE_WARPS + w) * (32 / G) + sub; it < total;
       it += ng) {
    const uint2 p = list[list_cap - 1 - it];
    const or_gallop_edge d = or_gallop_get(p, __ldg(sl + p.y), __ldg(vinfo + p.x));
    const uint32_t c = or_gallop_group<G>(dst, d.xb, d.xe, d.yb, d.ye, gl, gmask, cnt);
    if (gl == 0 && c) atomicAdd(cnt + d.at, (int32_t)c);
    if (gl == 0) found += c;
  }
  if (gl == 0 && found) atomicAdd(&ctr[C_MATCH + ACCX_KIND_GALLOP], found);
}

// A warp takes 32 edges, a lane loading each one's records (the next 32 edges' while these
// are walked).  Partner lists of up to GALLOP_LANE ids are the lane's own: both lists
// walked together, or the partner's ids searched where the owner's list is much longer;
// eight-lane groups take the longer ones.  A group for every edge spent ~25 warp
// instructions on two lists of ten ids; walking with a branch per advance, 34.  Erdos-
// Renyi with 16M entries 569 -> 330 us, with 120M, whose lists come from HBM,
// 3.60 -> 2.23 ms; R-MAT 24, with 58 ids a list, would take 12.7 ms instead of 10.1.
#define GALLOP_LANE 32u   // partner ids up to which a lane takes the edge alone
#define GALLOP_MERGE 8u   // owner ids per partner id up to which it walks both lists
// per SM: with more the partner lists push each other out of L1 (Erdos-Renyi with 120M
// entries: 4 CTAs 2.55 ms, 5 2.23, 6 2.46, 8 3.1; a prefetch of the next lists into L2 cost
// 0.6 ms)
#define GALLOP_CTAS 5
__global__ void __launch_bounds__(MERGE_WARPS * 32, GALLOP_CTAS) k_gallop_lane(const uint2 *__restrict__ vinfo,
                                                                                const int32_t *__restrict__ dst,
                                                                                const uint2 *__restrict__ sl,
                                                                                const uint2 *__restrict__ list,
                                                                                uint32_t list_cap,
                                                                                unsigned long long *__restrict__ ctr,
                                                                                int32_t *__restrict__ cnt) {
  if (or_gallop_long(ctr)) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, sub = lane / 8, gl = lane % 8;
  const unsigned gmask = 0xffu << (sub * 8);
  uint32_t found = 0;
  const uint32_t total = (uint32_t)(ctr[C_GALLOP] < list_cap ? ctr[C_GALLOP] : list_cap);
  const uint32_t step = gridDim.x * MERGE_WARPS * 32;
  auto load = [&](uint32_t it, uint2 *p) {
    *p = make_uint2(0u, 0u);
    if (it >= total) return false;
    *p = __ldg(list + (list_cap - 1 - it));
    return true;
  };
  uint32_t it = (blockIdx.x * MERGE_WARPS + w) * 32 + lane;
  uint2 p, r = make_uint2(0u, 0u), xi = make_uint2(0u, 0u);
  if (load(it, &p)) {
    r = __ldg(sl + p.y);
    xi = __ldg(vinfo + p.x);
  }
  for (uint32_t it0 = it - lane; it0 < total; it0 += step) {
    const or_gallop_edge d = or_gallop_get(p, r, xi);
    it = it0 + lane < 0xffffffffu - step ? it0 + lane + step : 0xffffffffu;
    if (load(it, &p)) {
      r = __ldg(sl + p.y);
      xi = __ldg(vinfo + p.x);
    } else {
      r = xi = make_uint2(0u, 0u);
    }
    const bool any = d.yb < d.ye && d.xb < d.xe, own = any && d.ye - d.yb <= GALLOP_LANE;
    if (own) {
      uint32_t c = 0;
      if (d.xe - d.xb <= GALLOP_MERGE * (d.ye - d.yb)) {
        // both ids loaded anew each step (mostly L1 hits; the array is padded past its
        // end): the only branches are the loop's and the rare match's
        uint32_t i = d.xb, j = d.yb;
        do {
          const int32_t a = __ldg(dst + i), b = __ldg(dst + j);
          if (a == b) {
            c++;
            atomicAdd(cnt + i, 1);
            atomicAdd(cnt + j, 1);
          }
          i += a <= b;
          j += b <= a;
        } while (i < d.xe && j < d.ye);
      } else {
        uint32_t lo = d.xb;
        for (uint32_t j = d.yb; j < d.ye && lo < d.xe; j++) {
          const int32_t id = __ldg(dst + j);
          lo = accx_lower_bound(dst, lo, d.xe, id);
          if (lo < d.xe && __ldg(dst + lo) == id) {
            c++;
            atomicAdd(cnt + lo, 1);
            atomicAdd(cnt + j, 1);
          }
        }
      }
      if (c) atomicAdd(cnt + d.at, (int32_t)c);
      found += c;
    }
    __syncwarp();
    for (unsigned big = __ballot_sync(ACCX_FULL_MASK, any && !own); big;) {
      // the group's edge: the sub-th of the next four
      unsigned m = big;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        if (q < sub) m &= m - 1;
        big &= big - 1;
      }
      const int src = m ? __ffs(m) - 1 : 0;
      const uint32_t gxb = __shfl_sync(ACCX_FULL_MASK, d.xb, src), exe = __shfl_sync(ACCX_FULL_MASK, d.xe, src);
      const uint32_t gyb = __shfl_sync(ACCX_FULL_MASK, d.yb, src), gye = __shfl_sync(ACCX_FULL_MASK, d.ye, src);
      const uint32_t gat = __shfl_sync(ACCX_FULL_MASK, d.at, src);
      const uint32_t c = or_gallop_group<8>(dst, gxb, m ? exe : gxb, gyb, gye, gl, gmask, cnt);
      if (gl == 0 && c) atomicAdd(cnt + gat, (int32_t)c);
      if (gl == 0) found += c;
      __syncwarp();
    }
  }
  unsigned long long f = found;
#pragma unroll
  for (int q = 16; q >= 1; q >>= 1) f += __shfl_xor_sync(ACCX_FULL_MASK, f, q);
  if (lane == 0 && f) atomicAdd(&ctr[C_MATCH + ACCX_KIND_GALLOP], f);
}

// Work items of the bitmap owners.  An owner with little probe work is one entry of
// the light list (a warp each, k_owner_warp); the others become items of the CTA
// kernel, cut into slices of about `target` probes.  items[] holds the CTA items from
// the front and the light owners from the back, slot[u] the first item of owner u.
// Together they never exceed n + m/32, as an owner has at most max(1, degree/32)
// slices.
//
// Light: at most OW_CAP prefix ids (the warp's table and counters), OW_DEG entries and
// OW_WORK probes -- up to OW_WORK_MAX on graphs whose owners average that much, so that
// many warps have several (all probes / OW_SPREAD), but no more than an OW_SHARE'th of all
// (a small graph's owners are fewer than the machine's warps).  A CTA spends ~4 us of
// staging and barriers on an item however small it is, a warp well under 1 us; with many
// probes one warp becomes the tail.  Counts (us) with 2048 / 4096 / 8192 / 16384: R-MAT 21
// 5949 / 5706 / 5362 / 5499, Chung-Lu 3M 3704 / 3523 / 3579 / 3914, R-MAT 18 602 / 590 / 627 /
// 628; without light owners a batch of 48 small graphs took 1929, with them 998.  Owners
// from a counter instead of a fixed stride: Chung-Lu 3M 3744.
//
// n here is the number of vertices that can own (ids below the dense window).  One
// cluster of eight CTAs counts and then fills in id order: the heavy owners come
// first, and neighbours in time share partner lists in L2 (slots handed out by
// atomics in a grid of 64 CTAs, about 16K ids out of order, cost the CTA kernel 1.3 %
// at R-MAT 24).  A count, device scan and fill over all n vertices were four launches,
// and one 64-bit atomic per owner for the owner-work statistic took 139 us of a
// 3M-vertex power-law count.
#define OW_CAP 512u
#define OW_SLOTS 1024u
#define OW_POS 11  // bits of a position in a table word; the ids, below the window, take the others
#define OW_WORK 4096u
#define OW_WORK_MAX 8192u
#define OW_SHARE 4096u
#define OW_SPREAD 400000u
#define OW_DEG 4096u
// CTA items aim at a 16th of a CTA's share of all probes, within these bounds (a
// smaller item costs its staging more often, a larger one ends later than the rest)
#define ITEM_TARGET_MIN 16384u
__device__ __forceinline__ uint32_t accx_item_target(const unsigned long long *__restrict__ ctr, uint32_t target_max,
                                                     uint32_t ctas) {
  const unsigned long long t = ctr[C_WORK + ACCX_KIND_BITMAP] / (16ull * ctas);
  return (uint32_t)(t < ITEM_TARGET_MIN ? ITEM_TARGET_MIN : t > target_max ? target_max : t);
}

__device__ __forceinline__ uint32_t accx_warp_incl_sum(uint32_t v, int lane) {
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t a = __shfl_up_sync(ACCX_FULL_MASK, v, d);
    if (lane >= d) v += a;
  }
  return v;
}

#define OI_CTAS 8
#define OI_THREADS 1024
#define OI_STEP 4  // vertices a lane takes at once: their loads are in flight together
// The CTA slices (0: none or light) of the vertices u0 + 32 r, r < OI_STEP, of this lane.
__device__ __forceinline__ void ow_shape(const uint32_t *__restrict__ off, const uint32_t *__restrict__ pre,
                                         const unsigned long long *__restrict__ work_u, uint32_t u0, uint32_t e,
                                         uint32_t target, uint32_t light_max, uint32_t (&ns)[OI_STEP],
                                         bool (&light)[OI_STEP], uint32_t (&px)[OI_STEP]) {
  unsigned long long w[OI_STEP];
  uint32_t du[OI_STEP];
#pragma unroll
  for (int r = 0; r < OI_STEP; r++) {
    const uint32_t u = u0 + 32u * r;
    w[r] = u < e ? work_u[u] : 0ull;
    du[r] = u < e ? __ldg(off + u + 1) - __ldg(off + u) : 0u;
    px[r] = u < e ? __ldg(pre + u) : 0u;
  }
#pragma unroll
  for (int r = 0; r < OI_STEP; r++) {
    light[r] = w[r] && px[r] <= OW_CAP && w[r] <= light_max && du[r] <= OW_DEG;
    uint32_t nc;
    ns[r] = 0;
    if (w[r] && !light[r]) accx_item_shape(du[r], 0, w[r], 1, target, &nc, &ns[r]);
  }
}

__global__ void __cluster_dims__(OI_CTAS, 1, 1) __launch_bounds__(OI_THREADS)
    k_owner_items(const uint32_t *__restrict__ off, const uint32_t *__restrict__ pre, uint32_t n,
                  const unsigned long long *__restrict__ work_u, uint32_t target_max, uint32_t ctas, uint32_t cap,
                  unsigned long long *__restrict__ slot, uint32_t *__restrict__ items,
                  unsigned long long *__restrict__ ctr) {
  __shared__ uint32_t s_h[32], s_l[32], s_tot[2];
  cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t target = accx_item_target(ctr, target_max, ctas);
  const unsigned long long share = ctr[C_WORK + ACCX_KIND_BITMAP] / OW_SHARE;
  const unsigned long long mean = ctr[C_WORK + ACCX_KIND_BITMAP] / OW_SPREAD;
  uint32_t light_max = mean < OW_WORK ? OW_WORK : mean > OW_WORK_MAX ? OW_WORK_MAX : (uint32_t)mean;
  if (share < light_max) light_max = (uint32_t)share;
  // a run of `span` vertices (a multiple of 32) per warp of the cluster
  const uint32_t nw = OI_CTAS * OI_THREADS / 32, span = ((n + nw - 1) / nw + 31u) & ~31u;
  const uint32_t b = min(n, (cl.block_rank() * (OI_THREADS / 32) + warp) * span), e = min(n, b + span);
  unsigned long long staged = 0;
  uint32_t h = 0, l = 0;
  for (uint32_t u0 = b; u0 < e; u0 += 32 * OI_STEP) {
    bool light[OI_STEP];
    uint32_t ns[OI_STEP], px[OI_STEP];
    ow_shape(off, pre, work_u, u0 + lane, e, target, light_max, ns, light, px);
#pragma unroll
    for (int r = 0; r < OI_STEP; r++) {
      h += ns[r];
      l += light[r];
      staged += (unsigned long long)px[r] * (light[r] ? 1u : ns[r]);
    }
  }
  h = __reduce_add_sync(ACCX_FULL_MASK, h);
  l = __reduce_add_sync(ACCX_FULL_MASK, l);
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) staged += __shfl_xor_sync(ACCX_FULL_MASK, staged, d);
  if (lane == 0) {
    if (staged) atomicAdd(&ctr[C_OWNER + ACCX_KIND_BITMAP], staged);
    s_h[warp] = h;
    s_l[warp] = l;
  }
  __syncthreads();
  if (warp == 0) {
    const uint32_t vh = s_h[lane], vl = s_l[lane];
    const uint32_t ih = accx_warp_incl_sum(vh, lane), il = accx_warp_incl_sum(vl, lane);
    s_h[lane] = ih - vh;
    s_l[lane] = il - vl;
    if (lane == 31) {
      s_tot[0] = ih;
      s_tot[1] = il;
    }
  }
  cl.sync();
  uint32_t h0 = s_h[warp], l0 = s_l[warp];
  for (unsigned r = 0; r < cl.block_rank(); r++) {
    const uint32_t *t = cl.map_shared_rank(s_tot, r);
    h0 += t[0];
    l0 += t[1];
  }
  if (cl.block_rank() == OI_CTAS - 1 && threadIdx.x == 0) {
    ctr[C_HEAVY] = h0 + s_tot[0];  // warp 0: the CTA's first slots
    ctr[C_LIGHT] = l0 + s_tot[1];
  }
  cl.sync();  // the totals are not read after this
  for (uint32_t u0 = b; u0 < e; u0 += 32 * OI_STEP) {
    bool light[OI_STEP];
    uint32_t ns[OI_STEP], px[OI_STEP];
    ow_shape(off, pre, work_u, u0 + lane, e, target, light_max, ns, light, px);
#pragma unroll
    for (int r = 0; r < OI_STEP; r++) {
      const uint32_t u = u0 + 32u * r + lane;
      const unsigned lm = __ballot_sync(ACCX_FULL_MASK, light[r]);
      const uint32_t incl = accx_warp_incl_sum(ns[r], lane), p = h0 + incl - ns[r];
      const uint32_t q = l0 + __popc(lm & ((1u << lane) - 1u));
      if (light[r] && q < cap) items[cap - 1 - q] = u;
      if (ns[r]) {
        slot[u] = p;
        for (uint32_t j = 0; j < ns[r] && p + j < cap; j++) items[p + j] = u;
      }
      h0 += __shfl_sync(ACCX_FULL_MASK, incl, 31);
      l0 += __popc(lm);
    }
  }
}

// Light bitmap owners: a warp per owner, no barriers.  The owner's prefix goes into
// a hash table of packed (id << OW_POS | position) words in the warp's shared memory
// (four slots an id up to 256 ids, so most look-ups read one word; at least two), with
// one counter per position; ids are below 2^21 as bitmap owners lie inside the window.  The
// row is walked 32 entries at a time: their partner ranges are concatenated (warp
// scan) and streamed 32 ids a step, four steps' loads in flight, as the CTA kernel
// streams its short lists.  Credits are the CTA kernel's.  Bound by latency and
// instruction issue.
#define OW_WARPS 8
struct ow_warp {
  uint32_t tab[OW_SLOTS];
  uint32_t oc[OW_CAP];
  uint32_t pre[33], beg[32], hit[32];
};

__device__ __forceinline__ uint32_t ow_hash(uint32_t id, int sh) { return (id * 0x9E3779B1u) >> sh; }

__global__ void __launch_bounds__(OW_WARPS * 32) k_owner_warp(const uint32_t *__restrict__ off,
                                                              const int32_t *__restrict__ dst,
                                                              const uint32_t *__restrict__ pre,
                                                              const uint32_t *__restrict__ items, uint32_t cap,
                                                              const uint2 *__restrict__ sl, int32_t *__restrict__ cnt,
                                                              unsigned long long *__restrict__ ctr) {
  extern __shared__ __align__(16) uint32_t smem[];
  const int lane = threadIdx.x & 31;
  ow_warp &S = reinterpret_cast<ow_warp *>(smem)[threadIdx.x >> 5];
  const uint32_t total = (uint32_t)(ctr[C_LIGHT] < cap ? ctr[C_LIGHT] : cap);
  unsigned long long found = 0;
  const uint32_t nw = gridDim.x * OW_WARPS;
  uint32_t it = blockIdx.x * OW_WARPS + (threadIdx.x >> 5);
  // a row is a chain of dependent loads: the next row's bounds, and this row's first ids
  // and ranges, are loaded ahead of where they are used
  uint32_t x = it < total ? items[cap - 1 - it] : 0u;
  uint32_t nb = it < total ? __ldg(off + x) : 0u, ne = it < total ? __ldg(off + x + 1) : 0u;
  uint32_t np = it < total ? __ldg(pre + x) : 0u;
  while (it < total) {
    const uint32_t ub = nb, ue = ne, px = min(np, OW_CAP);
    const uint32_t id0 = (uint32_t)lane < px ? (uint32_t)__ldg(dst + ub + lane) : 0u;
    uint2 sn = ub + lane < ue ? __ldg(sl + ub + lane) : make_uint2(0u, 0u);
    it += nw;
    const bool more = it < total;
    x = more ? items[cap - 1 - it] : 0u;
    // the table: 64 to 1024 slots
    int lg = 6;
    while (lg < 10 && (1u << lg) < 4u * px) lg++;
    const uint32_t mask = (1u << lg) - 1u;
    const int sh = 32 - lg;
    for (uint32_t i = lane; i <= mask; i += 32) S.tab[i] = 0xffffffffu;
    for (uint32_t i = lane; i < px; i += 32) S.oc[i] = 0;
    __syncwarp();
    for (uint32_t i = lane; i < px; i += 32) {
      const uint32_t id = i < 32 ? id0 : (uint32_t)__ldg(dst + ub + i);
      uint32_t h = ow_hash(id, sh);
      while (atomicCAS(&S.tab[h], 0xffffffffu, (id << OW_POS) | i) != 0xffffffffu) h = (h + 1) & mask;
    }
    __syncwarp();
    nb = more ? __ldg(off + x) : 0u;
    ne = more ? __ldg(off + x + 1) : 0u;
    np = more ? __ldg(pre + x) : 0u;
    for (uint32_t r0 = ub; r0 < ue; r0 += 32) {
      const uint32_t k = r0 + lane;
      const uint32_t sst = sn.x, len = (sn.y & OR_SL_GALLOP) ? 0u : sn.y;
      sn = k + 32 < ue ? __ldg(sl + k + 32) : make_uint2(0u, 0u);
      const unsigned act = __ballot_sync(ACCX_FULL_MASK, len > 0);
      if (!act) continue;
      const uint32_t incl = accx_warp_incl_sum(len, lane);
      const uint32_t tot = __shfl_sync(ACCX_FULL_MASK, incl, 31), nseg = __popc(act);
      const uint32_t me = __popc(act & ((1u << lane) - 1u));
      if (len) {
        S.pre[me] = incl - len;
        S.beg[me] = sst;
        S.hit[me] = 0;
      }
      if (lane == 0) S.pre[nseg] = tot;
      __syncwarp();
      uint32_t segb = 0;
      for (uint32_t c0 = 0; c0 < tot; c0 += 32u * PROBE_UNROLL) {
        int32_t xs[PROBE_UNROLL];
        uint32_t sg[PROBE_UNROLL], gi[PROBE_UNROLL];
#pragma unroll
        for (int r = 0; r < PROBE_UNROLL; r++) {
          // 32 ids meet at most 31 segment starts after segb: each lane loads one
          // start, and a lane's segment is segb + the starts at or before its id
          const uint32_t i0 = c0 + 32u * r, i = i0 + lane;
          const uint32_t kb = segb + 1u + lane;
          const uint32_t o = (kb <= nseg ? S.pre[kb] : 0xffffffffu) - i0;
          const unsigned M = __reduce_or_sync(ACCX_FULL_MASK, o < 32u ? (1u << o) : 0u);
          const uint32_t sj = min(segb + __popc(M & (0xffffffffu >> (31 - lane))), 31u);
          sg[r] = sj;
          gi[r] = (i < tot) ? S.beg[sj] + (i - S.pre[sj]) : 0u;
          xs[r] = (i < tot) ? __ldg(dst + gi[r]) : -1;
          segb += __popc(M) + (__ballot_sync(ACCX_FULL_MASK, o == 32u) ? 1u : 0u);
        }
#pragma unroll
        for (int r = 0; r < PROBE_UNROLL; r++) {
          if (xs[r] < 0) continue;
          const uint32_t id = (uint32_t)xs[r];
          uint32_t h = ow_hash(id, sh), t = S.tab[h];
          while ((t >> OW_POS) != id && t != 0xffffffffu) {
            h = (h + 1) & mask;
            t = S.tab[h];
          }
          if (t != 0xffffffffu) {
            atomicAdd(cnt + gi[r], 1);
            atomicAdd(&S.oc[t & ((1u << OW_POS) - 1u)], 1u);
            atomicAdd(&S.hit[sg[r]], 1u);
          }
        }
      }
      __syncwarp();
      if (len) {  // the edge's credit, to its prefix entry
        const uint32_t h = S.hit[me];
        found += h;
        if (h) {
          if (k - ub < px) atomicAdd(&S.oc[k - ub], h);
          else atomicAdd(cnt + sst + len, (int32_t)h);
        }
      }
      __syncwarp();
    }
    for (uint32_t i = lane; i < px; i += 32) {
      const uint32_t h = S.oc[i];
      if (h) atomicAdd(cnt + ub + i, (int32_t)h);
    }
    __syncwarp();
  }
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) found += __shfl_xor_sync(ACCX_FULL_MASK, found, d);
  if (lane == 0 && found) atomicAdd(&ctr[C_MATCH + ACCX_KIND_BITMAP], found);
}

// Dense rows: the triangles a < b < c of bitmap-kind edges with a among the first K
// ids (the hubs after the degree relabel) and c among the first M, counted a word at
// a time.  T[x] is a K-bit mask of P(x) ∩ [0, K) for every row x < M.  The row x of a
// triangle's b or c meets the other one, y, as a neighbour, so over all neighbours
// y < M of x
//   * sum over y of T[y], taken at the bits of T[x], is the number of these triangles
//     on the edge (x, a), for every hub a at once;
//   * popc(T[x] & T[y]), for y < x, is their number on the edge (x, y).
// The sums are kept as vertical (bit-sliced) counters: a lane holds K/1024 words of
// each of ten bit planes and adds a neighbour's word to 32 counters with about 2.3
// three-input logic operations (carry-save adders, 32 neighbours a round), so no
// common id is ever enumerated and nothing is credited by atomics until the row's
// end, where each of its entries below K takes its counter's value.  The list-probing
// kernels then start a partner's list behind its ids below K for these edges.
//
// Probing spent ~54 thread instructions an id (a hit costs a rank, a RED and a shared
// atomic); at R-MAT 24 the 61 % of all probes that lie on edges with c < 65536 have
// 65-98 % of their ids below 4096.  K and M come from k_dense_plan.  Measured at
// R-MAT 24 (K 4096, M 131072): list probing 71.2 -> 39.6 ms for 8.6 ms here; Chung-Lu 3M:
// 4.2 -> 2.4 ms for both.
#define DENSE_PLANES 10   // bits of a counter: it takes every neighbour of an item
#define DENSE_WARPS 8

// T, low[x] = |T[x]| and the work items of the rows below M: a warp per row.
// item = (row, first entry, entries), at most `chunk` entries below M of the row.
template <int WPL>
__global__ void __launch_bounds__(256) k_dense_rows(const uint32_t *__restrict__ off, const int32_t *__restrict__ dst,
                                                    const uint32_t *__restrict__ pre, uint32_t M, uint32_t chunk,
                                                    uint32_t *__restrict__ T, uint32_t *__restrict__ low,
                                                    uint4 *__restrict__ items, uint32_t cap,
                                                    unsigned long long *__restrict__ nitems) {
  constexpr uint32_t K = WPL * 1024u;
  __shared__ uint32_t s_t[8][WPL * 32];
  const int lane = threadIdx.x & 31;
  uint32_t *t = s_t[threadIdx.x >> 5];
  const uint32_t nw = gridDim.x * 8u;
  for (uint32_t x = blockIdx.x * 8u + (threadIdx.x >> 5); x < M; x += nw) {
    const uint32_t b = off[x], px = pre[x];
#pragma unroll
    for (int k = 0; k < WPL; k++) t[k * 32 + lane] = 0;
    __syncwarp();
    uint32_t lw = 0;
    for (uint32_t i0 = 0; i0 < px; i0 += 32) {
      const uint32_t id = i0 + lane < px ? (uint32_t)__ldg(dst + b + i0 + lane) : 0xffffffffu;
      if (id < K) atomicOr(&t[id >> 5], 1u << (id & 31u));
      const unsigned in = __ballot_sync(ACCX_FULL_MASK, id < K);
      lw += __popc(in);
      if (in != ACCX_FULL_MASK) break;
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < WPL; k++) T[(size_t)x * (WPL * 32) + k * 32 + lane] = t[k * 32 + lane];
    if (lane == 0) {
      low[x] = lw;
      if (lw) {
        const uint32_t e = off[x + 1], c = accx_lower_bound(dst, b, e, (int32_t)M) - b;
        const uint32_t nch = (c + chunk - 1) / chunk;
        const unsigned long long p = atomicAdd(nitems, (unsigned long long)nch);
        for (uint32_t j = 0; j < nch && p + j < cap; j++)
          items[p + j] = make_uint4(x, b + j * chunk, min(chunk, c - j * chunk), 0u);
      }
    }
    __syncwarp();
  }
}

// full adder on 32 counters' bits: l += a + b, the carries to h
__device__ __forceinline__ void accx_csa(uint32_t &h, uint32_t &l, uint32_t a, uint32_t b) {
  h = (l & a) | (l & b) | (a & b);
  l = l ^ a ^ b;
}

// The masks of eight neighbours (lanes g0..g0+7 of y, the set ones of act) on their
// way into shared memory, one asynchronous copy of 4 WPL bytes a lane and row; rows that
// are not active, and words past the smaller of x and y (no triangle there), arrive as
// zeros without a read.
template <int WPL>
__device__ __forceinline__ void dense_issue(uint32_t sbuf, const uint32_t *__restrict__ T, uint32_t x, uint32_t y,
                                            unsigned act, int g0, int lane) {
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const uint32_t yi = __shfl_sync(ACCX_FULL_MASK, y, g0 + i);
    const bool in = ((act >> (g0 + i)) & 1u) && (uint32_t)lane * (WPL * 32) < min(x, yi);
    const uint32_t *src = T + (in ? (size_t)yi * (WPL * 32) + lane * WPL : 0);
    const int bytes = in ? WPL * 4 : 0;
    const uint32_t to = sbuf + (uint32_t)(i * 32 + lane) * (WPL * 4);
    if (WPL == 4)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(src), "r"(bytes) : "memory");
    else if (WPL == 2)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(to), "l"(src), "r"(bytes) : "memory");
    else
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(to), "l"(src), "r"(bytes) : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

template <int WPL>
__device__ __forceinline__ void dense_read(uint32_t (&w)[WPL], const uint32_t *p) {
  if (WPL == 4) {
    const uint4 q = *reinterpret_cast<const uint4 *>(p);
    w[0] = q.x; w[1 % WPL] = q.y; w[2 % WPL] = q.z; w[3 % WPL] = q.w;
  } else if (WPL == 2) {
    const uint2 q = *reinterpret_cast<const uint2 *>(p);
    w[0] = q.x; w[1 % WPL] = q.y;
  } else {
    w[0] = *p;
  }
}

// Eight neighbours' masks into the low planes; the carries of weight eight to e8.  POP:
// also popc(T[x] & T[y]), kept by the lane of y in `pc` (two sums to a warp reduction:
// each is at most 4096).
template <int WPL, bool POP>
__device__ __forceinline__ void dense_eight(const uint32_t *buf, int g0, int lane, const uint32_t (&tx)[WPL],
                                            uint32_t (&pl)[DENSE_PLANES][WPL], uint32_t (&e8)[WPL], uint32_t &pc) {
  uint32_t w[8][WPL];
#pragma unroll
  for (int i = 0; i < 8; i++) dense_read<WPL>(w[i], buf + (i * 32 + lane) * WPL);
  if (POP) {
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      uint32_t c = 0, d = 0;
#pragma unroll
      for (int k = 0; k < WPL; k++) {
        c += __popc(w[i][k] & tx[k]);
        d += __popc(w[i + 1][k] & tx[k]);
      }
      c = __reduce_add_sync(ACCX_FULL_MASK, c + (d << 16));
      if (lane == g0 + i) pc = c & 0xffffu;
      if (lane == g0 + i + 1) pc = c >> 16;
    }
  }
#pragma unroll
  for (int k = 0; k < WPL; k++) {
    uint32_t ta, tb, fa, fb;
    accx_csa(ta, pl[0][k], w[0][k], w[1][k]);
    accx_csa(tb, pl[0][k], w[2][k], w[3][k]);
    accx_csa(fa, pl[1][k], ta, tb);
    accx_csa(ta, pl[0][k], w[4][k], w[5][k]);
    accx_csa(tb, pl[0][k], w[6][k], w[7][k]);
    accx_csa(fb, pl[1][k], ta, tb);
    accx_csa(e8[k], pl[2][k], fa, fb);
  }
}

// A warp per item.  The neighbours' masks come through a ring of two groups of eight in
// the warp's shared memory: the next group is copied while this one is added, so the
// loads in flight do not cost registers (R-MAT 24 count 70.7 -> 69.2 ms against loads
// into registers; three CTAs an SM instead of two spill at K 4096: 70.0).  The ALU pipe
// is the busiest (60 %), L2 at a third of its peak.  ALL: every edge between rows below
// M is of the bitmap kind; otherwise each neighbour's kind is looked up as classify
// does.
template <int WPL>
struct dense_ring {
  uint32_t w[2][8 * 32 * WPL];  // also takes the planes at the item's end: DENSE_PLANES x 32 WPL words
};
template <int WPL, bool ALL>
__global__ void __launch_bounds__(DENSE_WARPS * 32, 2) k_dense_pairs(
    const uint32_t *__restrict__ off, const int32_t *__restrict__ dst, const uint32_t *__restrict__ pre,
    const uint32_t *__restrict__ low, const uint32_t *__restrict__ T, const uint4 *__restrict__ items, uint32_t cap,
    const unsigned long long *__restrict__ nitems, int policy, const uint8_t *__restrict__ table, uint32_t pcap, int32_t *__restrict__ cnt,
    unsigned long long *__restrict__ ctr) {
  static_assert(DENSE_PLANES <= 16, "planes fit the ring");
  extern __shared__ __align__(16) uint32_t smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t *ring = reinterpret_cast<dense_ring<WPL> *>(smem)[warp].w[0];
  const uint32_t sring = (uint32_t)__cvta_generic_to_shared(ring);
  constexpr uint32_t GROUP = 8 * 32 * WPL;  // words of a group
  unsigned long long total = *nitems;
  if (total > cap) total = cap;
  unsigned long long found = 0;
  const unsigned long long nw = (unsigned long long)gridDim.x * DENSE_WARPS;
  for (unsigned long long it = (unsigned long long)blockIdx.x * DENSE_WARPS + warp; it < total; it += nw) {
    const uint4 item = __ldg(items + it);
    const uint32_t x = item.x, eb = item.y, ec = item.z;
    const uint32_t px = ALL ? 0u : __ldg(pre + x);
    uint32_t tx[WPL], pl[DENSE_PLANES][WPL];
    dense_read<WPL>(tx, T + (size_t)x * (WPL * 32) + lane * WPL);
#pragma unroll
    for (int p = 0; p < DENSE_PLANES; p++)
#pragma unroll
      for (int k = 0; k < WPL; k++) pl[p][k] = 0;
    auto active = [&](uint32_t y) {
      bool on = y != 0xffffffffu;
      if (!ALL && on) on = accx_dense_edge(policy, table, x, px, y, __ldg(pre + y), pcap);
      return __ballot_sync(ACCX_FULL_MASK, on);
    };
    uint32_t y = (uint32_t)lane < ec ? (uint32_t)__ldg(dst + eb + lane) : 0xffffffffu;
    uint32_t yn = 32u + lane < ec ? (uint32_t)__ldg(dst + eb + 32 + lane) : 0xffffffffu;
    unsigned act = active(y);
    dense_issue<WPL>(sring, T, x, y, act, 0, lane);
    for (uint32_t j = 0; j < ec; j += 32) {
      const unsigned actn = active(yn);
      const unsigned below = __ballot_sync(ACCX_FULL_MASK, y < x) & act;
      uint32_t pc = 0;
      uint32_t e8[4][WPL];
#pragma unroll
      for (int g = 0; g < 4; g++) {
        // the next group on its way (at the end of the row: an empty one), then this one
        if (g < 3) dense_issue<WPL>(sring + ((g + 1) & 1) * GROUP * 4, T, x, y, act, 8 * (g + 1), lane);
        else dense_issue<WPL>(sring, T, x, yn, actn, 0, lane);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        const uint32_t *buf = ring + (g & 1) * GROUP;
        if ((below >> (8 * g)) & 0xffu) {
          dense_eight<WPL, true>(buf, 8 * g, lane, tx, pl, e8[g], pc);
        } else if ((act >> (8 * g)) & 0xffu) {
          dense_eight<WPL, false>(buf, 8 * g, lane, tx, pl, e8[g], pc);
        } else {
#pragma unroll
          for (int k = 0; k < WPL; k++) e8[g][k] = 0;
        }
        __syncwarp();
      }
#pragma unroll
      for (int k = 0; k < WPL; k++) {
        uint32_t a, b, c;
        accx_csa(a, pl[3][k], e8[0][k], e8[1][k]);
        accx_csa(b, pl[3][k], e8[2][k], e8[3][k]);
        accx_csa(c, pl[4][k], a, b);
#pragma unroll
        for (int p = 5; p < DENSE_PLANES; p++) {
          const uint32_t o = pl[p][k];
          pl[p][k] = o ^ c;
          c &= o;
        }
      }
      if (((below >> lane) & 1u) && pc) {
        found += pc;
        atomicAdd(cnt + eb + j + lane, (int32_t)pc);
      }
      y = yn;
      act = actn;
      yn = j + 64 + lane < ec ? (uint32_t)__ldg(dst + eb + j + 64 + lane) : 0xffffffffu;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    // the counters of the row's hub entries, through shared memory
#pragma unroll
    for (int p = 0; p < DENSE_PLANES; p++)
#pragma unroll
      for (int k = 0; k < WPL; k++) ring[p * (WPL * 32) + lane * WPL + k] = pl[p][k];
    __syncwarp();
    const uint32_t ub = __ldg(off + x), lw = __ldg(low + x);
    for (uint32_t i = lane; i < lw; i += 32) {
      const uint32_t a = (uint32_t)__ldg(dst + ub + i), wd = (a >> 5) & (WPL * 32 - 1), bit = a & 31u;
      uint32_t v = 0;
#pragma unroll
      for (int p = 0; p < DENSE_PLANES; p++) v |= ((ring[p * (WPL * 32) + wd] >> bit) & 1u) << p;
      if (v) atomicAdd(cnt + ub + i, (int32_t)v);
    }
    __syncwarp();
  }
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) found += __shfl_xor_sync(ACCX_FULL_MASK, found, d);
  if (lane == 0 && found) atomicAdd(&ctr[C_MATCH + ACCX_KIND_BITMAP], found);
}

// One piece of a long list for one warp: G pair groups (64 G ids) from the
// even entry j0.  Lane pairs (j, j+1) come from one 8-byte load; ids outside
// [a0, a1) are dropped (the array's padding keeps the last pair in bounds).
// Every load is issued before the probes (a test per load would serialise
// them); the probes stop at the first pair group past the list end.  A hit at
// entry j credits cnt[j] -- a warp's credits for one load land in one line of
// cnt -- and the owner counter of the id's rank; returns this lane's hits.
template <int G>
__device__ __forceinline__ uint32_t or_piece(const int32_t *__restrict__ dst, uint32_t j0, uint32_t a0, uint32_t a1,
                                             uint32_t lane, uint32_t W, const uint32_t *words, const uint16_t *wbase,
                                             uint32_t *ocnt, uint32_t pxs, int32_t *__restrict__ cnt) {
  const uint32_t rem = a1 - j0;
  int2 v[G];
#pragma unroll
  for (int r = 0; r < G; r++) {
    const uint32_t j = j0 + 64u * r + 2u * lane;
    v[r] = j < a1 ? __ldg(reinterpret_cast<const int2 *>(dst + j)) : make_int2(-1, -1);
    if (j < a0) v[r].x = -1;
    if (j + 1u >= a1) v[r].y = -1;
  }
  int32_t *const cl = cnt + j0 + 2u * lane;
  uint32_t h = 0;
#pragma unroll
  for (int r = 0; r < 2 * G; r++) {
    if (64u * (uint32_t)(r >> 1) >= rem) break;
    const uint32_t id = min((uint32_t)((r & 1) ? v[r >> 1].y : v[r >> 1].x), W);  // W: the zero word
    const uint32_t wd = words[id >> 5];
    if ((wd >> (id & 31u)) & 1u) {
      // the rank: the word's base plus the set bits up to and including this one, less one
      const uint32_t rk = wbase[id >> 5] + __popc(wd << (~id & 31u)) - 1u;
      h++;
      atomicAdd(cl + 64u * (r >> 1) + (uint32_t)(r & 1), 1);
      atomicAdd(&ocnt[rk], 1u);  // rk < pxs on a sorted CSR, < pxs + 31 always (spare counters)
    }
  }
  return h;
}

#define LONG_PIECE (32u * LONG_UNROLL)    // ids per piece of a long list

// Bitmap kind.  CTAs take work items (an owner x, or a slice of its list when the
// owner's probe work is large) from a device counter.  The owner's prefix -- ids below
// x, which the classifier keeps below W -- is staged as a dense bitmap over [0, W)
// plus, per non-empty 32-bit word, the prefix position of the word's first id (rank of
// an id = that base + popcount of the lower bits).  The warps then take the slice's
// entries a ticket (at most 32) at a time from a shared queue and need no barrier until its end: the
// classifier stored, per bitmap entry (x,y), where P(y) starts and its length cut at
// min(x,y) (0 for other entries), one coalesced load.  A long probe list is walked by
// the whole warp in pieces of LONG_PIECE ids, its bounds and hits staying in registers;
// short ones are concatenated (warp scan) and streamed 32 ids a step.  A hit at partner
// entry j credits cnt[j] (RED), the owner's shared counter of the id's rank, and the
// edge (after the 32 entries).
// NT = the largest block size (blockDim.x <= NT); four 256-thread CTAs an SM with the
// default window, two of 512 threads with windows up to ~60 KiB.
// Bound by instruction issue and latency.  The earlier form took rounds of blockDim
// entries with CTA scans and four barriers each, and one queue entry per long list:
// ~0.15 ns a list and 0.84 ps an id at R-MAT 22 and 24 (R-MAT 24 count 69.2 -> 64.0 ms,
// Chung-Lu 3M 4.12 -> 3.90).
// A ticket is 32 entries of a long item, fewer of a short one, so that every warp gets four:
// with 32 always, the items of graphs with long lists and short rows, down to 32 entries,
// were one warp's work (counts, us, earlier form / 32 always / now: 3000 vertices of degree 850
// in their own numbering 700 / 924 / 652, 100 cliques of 200 relabeled 558 / 607 / 473, with
// 1024 threads 955 / 1457 / 602; R-MAT 22 12.4 -> 11.7 ms; two tickets a warp 11.8, one 12.4).
// A ticket with more than four warps' share of the item's probes in long lists leaves them to
// all warps, after a barrier that other items do without (vertices joined to all of 2000 hubs
// and to a few of each other, in their own numbering: 279 / 478 / 274; R-MAT 24 +0.6 %).
struct or_seg {
  uint32_t pre[33], beg[32], hit[32];
};
#define TICKET_MIN 4u     // entries of the smallest ticket
#define TICKETS_PER 4u    // tickets a warp that an item is cut into, if they are 32 entries at most
#define LEFT_CAP 64u      // lists that an item leaves to all warps
template <int NT>
__global__ void __launch_bounds__(NT, 1024 / NT) k_bitmap_or(const uint32_t *__restrict__ off,
                                                       const int32_t *__restrict__ dst,
                                                       const uint32_t *__restrict__ pre,
                                                       const uint32_t *__restrict__ items, uint32_t items_cap,
                                                       const unsigned long long *__restrict__ work_u,
                                                       const unsigned long long *__restrict__ slot,
                                                       const uint2 *__restrict__ sl, uint32_t W, uint32_t pcap,
                                                       uint32_t target_max, int32_t *__restrict__ cnt,
                                                       unsigned long long *__restrict__ ctr) {
  extern __shared__ __align__(16) uint32_t smem[];
  const uint32_t nwords = W / 32;
  uint32_t *words = smem;                                          // nwords + a zero word (ids >= W probe it)
  // pcap owner-prefix counters + 32 spares: a found id's rank is at most a word's
  // base (< pxs) + 31, so the counter add needs no bounds test even on unsorted input
  uint32_t *ocnt = smem + nwords + 4;
  uint16_t *wbase = reinterpret_cast<uint16_t *>(ocnt + pcap + 32);  // nwords first-id positions
  __shared__ or_seg s_seg[NT / 32];
  // the next item, fetched while the current one is walked: x, its first and last entry
  // to walk, row start, prefix length and probes (x = 0xffffffff: none)
  __shared__ uint32_t s_item[6], s_next;
  __shared__ uint4 s_left[LEFT_CAP];  // (first entry, end, edge) of lists left to all warps
  __shared__ uint32_t s_lists, s_taken;
  const int tid = threadIdx.x, nt = blockDim.x;
  const int lane = tid & 31;
  or_seg &S = s_seg[tid >> 5];
  auto fetch = [&]() {
    unsigned long long total = ctr[C_HEAVY];
    if (total > items_cap) total = items_cap;
    const unsigned long long it = atomicAdd(&ctr[C_ITEMS], 1ull);
    uint32_t x = 0xffffffffu;
    if (it < total) {
      x = items[it];
      const uint32_t ub = off[x], du = off[x + 1] - ub;
      uint32_t nchunks, nsplit;
      accx_item_shape(du, 0, work_u[x], 1, accx_item_target(ctr, target_max, gridDim.x), &nchunks, &nsplit);
      const uint32_t sp = (uint32_t)(it - slot[x]);
      s_item[1] = ub + (uint32_t)((unsigned long long)du * sp / nsplit);
      s_item[2] = ub + (uint32_t)((unsigned long long)du * (sp + 1) / nsplit);
      s_item[3] = ub;
      s_item[4] = pre[x];
      s_item[5] = (uint32_t)min(work_u[x] / nsplit, 0xffffffffull);
    }
    s_item[0] = x;
  };
  for (uint32_t i = tid; i <= nwords; i += nt) words[i] = 0;
  unsigned long long found = 0;  // this thread's share, summed per warp at the end
  if (tid == 0) fetch();
  __syncthreads();
  for (;;) {
    const uint32_t x = s_item[0], pa = s_item[1], pb = s_item[2], ub = s_item[3], px = s_item[4];
    const uint32_t heavy = s_item[5] / max((uint32_t)nt >> 7, 1u);  // four warps' even share of the probes
    if (x == 0xffffffffu) break;
    const uint32_t pxs = px <= pcap ? px : 0;  // the classifier guarantees px <= pcap for bitmap owners
    for (uint32_t i = tid; i < pxs; i += nt) {
      const uint32_t id = (uint32_t)__ldg(dst + ub + i);
      if (id < W) {
        atomicOr(&words[id >> 5], 1u << (id & 31));
        if (i == 0 || ((uint32_t)__ldg(dst + ub + i - 1) >> 5) != (id >> 5)) wbase[id >> 5] = (uint16_t)i;
      }
      ocnt[i] = 0;
    }
    if (tid == 0) s_next = s_lists = s_taken = 0;
    __syncthreads();
    if (tid == 0) fetch();  // read by all after this item's last barrier
    __syncwarp();
    const uint32_t tk = min(32u, max(TICKET_MIN, (pb - pa) / (TICKETS_PER * ((uint32_t)nt >> 5))));
    for (;;) {
      uint32_t r0 = 0;
      if (lane == 0) r0 = atomicAdd(&s_next, tk);
      r0 = __shfl_sync(ACCX_FULL_MASK, r0, 0);
      if (r0 >= pb - pa) break;
      r0 += pa;
      const uint32_t k = r0 + (uint32_t)lane;
      uint32_t sst = 0, len = 0;
      if ((uint32_t)lane < tk && k < pb) {
        const uint2 e = sl[k];
        sst = e.x;
        len = (e.y & OR_SL_GALLOP) ? 0u : e.y;  // galloping entries are not this kernel's
      }
      uint32_t hits = 0;
      unsigned lm = __ballot_sync(ACCX_FULL_MASK, len >= LONG_SEG);
      if (lm & (lm - 1)) {
        if (__reduce_add_sync(ACCX_FULL_MASK, len >= LONG_SEG ? min(len, 1u << 26) : 0u) > heavy) {
          // all warps take these after the last ticket
          uint32_t p = 0;
          if (lane == 0) p = atomicAdd(&s_lists, (uint32_t)__popc(lm));
          p = __shfl_sync(ACCX_FULL_MASK, p, 0) + __popc(lm & ((1u << lane) - 1u));
          if (len >= LONG_SEG && p < LEFT_CAP) s_left[p] = make_uint4(sst, sst + len, k, 0u);
          lm = __ballot_sync(ACCX_FULL_MASK, len >= LONG_SEG && p >= LEFT_CAP);
        }
      }
      for (; lm; lm &= lm - 1) {
        // a long list, walked in pieces of LONG_PIECE ids from the even entry at or
        // before its start
        const int src = __ffs(lm) - 1;
        const uint32_t a0 = __shfl_sync(ACCX_FULL_MASK, sst, src);
        const uint32_t a1 = a0 + __shfl_sync(ACCX_FULL_MASK, len, src);
        uint32_t h = 0;
        for (uint32_t j0 = a0 & ~1u; j0 < a1; j0 = accx_entry_step(j0, LONG_PIECE, a1)) {
          // the last piece loads only the pair groups it needs (the size class is
          // warp-uniform, and each class issues all its loads at once)
          const uint32_t rem = a1 - j0;
          if (rem > 256u) h += or_piece<LONG_UNROLL / 2>(dst, j0, a0, a1, lane, W, words, wbase, ocnt, pxs, cnt);
          else if (rem > 128u) h += or_piece<4>(dst, j0, a0, a1, lane, W, words, wbase, ocnt, pxs, cnt);
          else if (rem > 64u) h += or_piece<2>(dst, j0, a0, a1, lane, W, words, wbase, ocnt, pxs, cnt);
          else h += or_piece<1>(dst, j0, a0, a1, lane, W, words, wbase, ocnt, pxs, cnt);
        }
        h = __reduce_add_sync(ACCX_FULL_MASK, h);
        if (lane == src) hits = h;
      }
      const bool is_short = len > 0 && len < LONG_SEG;
      const unsigned bs = __ballot_sync(ACCX_FULL_MASK, is_short);
      if (bs) {
        const uint32_t incl = accx_warp_incl_sum(is_short ? len : 0u, lane);
        const uint32_t tot = __shfl_sync(ACCX_FULL_MASK, incl, 31), nseg = __popc(bs);
        const uint32_t me = __popc(bs & ((1u << lane) - 1u));
        if (is_short) {
          S.pre[me] = incl - len;
          S.beg[me] = sst;
          S.hit[me] = 0;
        }
        if (lane == 0) S.pre[nseg] = tot;
        __syncwarp();
        uint32_t segb = 0;
        for (uint32_t c0 = 0; c0 < tot; c0 += 32u * PROBE_UNROLL) {
          int32_t xs[PROBE_UNROLL];
          uint32_t sg[PROBE_UNROLL], gi[PROBE_UNROLL];
#pragma unroll
          for (int r = 0; r < PROBE_UNROLL; r++) {
            // 32 ids meet at most 31 segment starts after segb: each lane loads one
            // start, and a lane's segment is segb + the starts at or before its id
            const uint32_t i0 = c0 + 32u * r, i = i0 + (uint32_t)lane;
            const uint32_t kb = segb + 1u + (uint32_t)lane;
            const uint32_t o = (kb <= nseg ? S.pre[kb] : 0xffffffffu) - i0;
            const unsigned M = __reduce_or_sync(ACCX_FULL_MASK, o < 32u ? (1u << o) : 0u);
            const uint32_t sj = min(segb + __popc(M & (0xffffffffu >> (31 - lane))), 31u);
            sg[r] = sj;
            gi[r] = (i < tot) ? S.beg[sj] + (i - S.pre[sj]) : 0u;
            xs[r] = (i < tot) ? __ldg(dst + gi[r]) : -1;
            segb += __popc(M) + (__ballot_sync(ACCX_FULL_MASK, o == 32u) ? 1u : 0u);
          }
#pragma unroll
          for (int r = 0; r < PROBE_UNROLL; r++) {
            // ids >= W (the -1 of lanes past the end) read the zero word
            const uint32_t id = min((uint32_t)xs[r], W);
            const uint32_t wd = words[id >> 5];
            if ((wd >> (id & 31u)) & 1u) {
              const uint32_t rk = wbase[id >> 5] + __popc(wd << (~id & 31u)) - 1u;
              atomicAdd(cnt + gi[r], 1);
              atomicAdd(&ocnt[rk], 1u);  // rk < pxs on a sorted CSR, < pxs + 31 always (spare counters)
              atomicAdd(&S.hit[sg[r]], 1u);
            }
          }
        }
        __syncwarp();
        if (is_short) hits = S.hit[me];
        __syncwarp();
      }
      // edge credits go to the edge's prefix entry: the entry itself when y < x
      // (through the owner's counters), else x's position in N(y), which is where the
      // partner range was cut
      found += hits;
      if (hits) {
        if (k - ub < pxs) atomicAdd(&ocnt[k - ub], hits);
        else atomicAdd(cnt + (k - ub < px ? k : sst + len), (int32_t)hits);
      }
    }
    __syncthreads();
    if (s_lists) {
      for (;;) {
        uint32_t i = 0;
        if (lane == 0) i = atomicAdd(&s_taken, 1u);
        i = __shfl_sync(ACCX_FULL_MASK, i, 0);
        if (i >= min(s_lists, LEFT_CAP)) break;
        const uint4 q = s_left[i];
        uint32_t h = 0;
        for (uint32_t j0 = q.x & ~1u; j0 < q.y; j0 = accx_entry_step(j0, 64u * 4u, q.y))
          h += or_piece<4>(dst, j0, q.x, q.y, lane, W, words, wbase, ocnt, pxs, cnt);
        h = __reduce_add_sync(ACCX_FULL_MASK, h);
        if (lane == 0 && h) {
          found += h;
          if (q.z - ub < pxs) atomicAdd(&ocnt[q.z - ub], h);
          else atomicAdd(cnt + (q.z - ub < px ? q.z : q.y), (int32_t)h);
        }
      }
      __syncthreads();
    }
    // owner-side credits to HBM, then clear what was staged
    for (uint32_t i = tid; i < pxs; i += nt) {
      const uint32_t h = ocnt[i];
      if (h) atomicAdd(cnt + ub + i, (int32_t)h);
    }
    const uint32_t span = min(nwords, x / 32u + 1u);
    if (span <= pxs) {
      for (uint32_t i = tid; i < span; i += nt) words[i] = 0;
    } else {
      for (uint32_t i = tid; i < pxs; i += nt) {
        const uint32_t id = (uint32_t)__ldg(dst + ub + i);
        if (id < W) words[id >> 5] = 0;
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) found += __shfl_xor_sync(ACCX_FULL_MASK, found, d);
  if (lane == 0 && found) atomicAdd(&ctr[C_MATCH + ACCX_KIND_BITMAP], found);
}

// Every credit lands on an edge's prefix entry (the entry in the larger id's
// list), which starts at the bias (written by classify); the other entry copies
// it.  One thread per entry: a suffix entry e = (v,u), u > v, takes the count of its
// reverse rev[e] > e (u's prefix entry); entries without a reverse (asymmetric
// input) keep the bias.
__global__ void k_combine_or(uint32_t m, const uint32_t *__restrict__ rev, int32_t *__restrict__ cnt) {
  const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= m) return;
  const uint32_t r = rev[e];
  if (r != 0xffffffffu && r > e) cnt[e] = cnt[r];
}

