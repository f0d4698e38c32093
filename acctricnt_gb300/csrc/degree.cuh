// The default policy's counts on a CSR known to be symmetric: the ratio-50 rule still
// says which kind an edge is of (and the statistics follow it), but the intersections
// themselves are done by a better algorithm than one list merge per edge.
//
// Large graphs: triangles on degree-ordered prefixes, without renumbering anything.
// F(x) = the neighbours of x that come before x in the order (degree descending, id);
// at most sqrt(2m) ids.  Every triangle is met once, on the edge of its two later
// vertices, as an id common to their F, and credited to its three edges; this is the
// oriented count (orient.cuh) with the order computed on the fly instead of a
// relabeled copy.  The vertex with the longer F owns the edge: it is staged, the other
// one's ids are streamed, so the credits of the busy hub edges stay in shared counters.
// Merging full lists up to a ratio of 50 cost 18.5 ms of an R-MAT 18 count: 19.4 -> 1.31
// ms (14.8x); power law with 4.6M entries 7.0 -> 0.61 ms.
//
// Small graphs: one kernel, a warp per owned edge (k_count_small).
//
// Included by count.cu.
#pragma once

// Entries up to which one kernel does it all.  That kernel / the degree-ordered count
// (us): R-MAT with 100K entries 63 / 85, with 200K 114 / 100; power law with 120K 58 / 86,
// with 240K 113 / 101; Erdos-Renyi with 120K 40 / 47, with 240K 68 / 49.
#define DG_SMALL_M (1u << 17)
// Rows above `row` entries are filtered and walked by CTAs, the others by warps: 64 on
// graphs of less than 2M entries, where one warp's row is the tail (R-MAT with 400K
// entries 131 us against 163 with 128), else 128 (R-MAT 18 1306 us against 1340).
#define DG_ROW_SMALL 64u
#define DG_ROW 128u
#define DG_ROW_M (1u << 21)
#define DG_SLICE 1024u         // entries of a row a CTA walks as one item
#define DG_LIGHT 32u           // |F| up to which a warp walks a row where it finds it
#define DG_TINY 4u             // |F| up to which a lane does, if the row has at most
#define DG_TINY_ROW 16u        // this many entries
#define DG_WARP 128u           // |F| a warp's table takes: listed rows
#define DG_KEEP 1024u          // list entries a CTA gathers before one atomic places them
#define DG_CAP 1024u           // |F| staged at once by a CTA
#define DG_SLOTS 4096u
#define DG_THREADS 256
// Rows above two tiles are cut at the entry tiles' ends and filtered by a CTA a piece: the keepers of
// each piece are counted first (k_dg_rows), so that a piece knows where its part of F begins.
// A CTA a row spent 1.5 us on 1024 entries: a star of 16M leaves took 25.1 ms (7.5 by an
// intersection per edge), now 2.5; of 100K leaves 126 us (92), now 64.
#define DG_TILE 8192u

// Per-kind statistics of an edge whose larger degree is dl, the smaller ds.
__device__ __forceinline__ void dg_stat(cl_stats &st, uint32_t dl, uint32_t ds) {
  st.add(accx_edge_kind(ACCX_POLICY_HEURISTIC, nullptr, dl, ds), ds, dl);
}
// Adds every thread's statistics to the counters (all threads of the CTA).
__device__ __forceinline__ void dg_stat_flush(const cl_stats &st, unsigned long long *s_st,
                                              unsigned long long *__restrict__ ctr) {
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < 9) s_st[threadIdx.x] = 0;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 2; k++) {  // merge and galloping
    const unsigned long long v[3] = {st.e[k], st.w[k], st.o[k]};
#pragma unroll
    for (int q = 0; q < 3; q++) {
      unsigned long long x = v[q];
#pragma unroll
      for (int d = 16; d >= 1; d >>= 1) x += __shfl_xor_sync(ACCX_FULL_MASK, x, d);
      if (lane == 0 && x) atomicAdd(&s_st[q * ACCX_NUM_KINDS + k], x);
    }
  }
  __syncthreads();
  if (threadIdx.x < 9 && s_st[threadIdx.x]) atomicAdd(&ctr[C_EDGES + threadIdx.x], s_st[threadIdx.x]);
}

// Does neighbour v (degree dv) come before u (degree du)?
__device__ __forceinline__ bool dg_before(uint32_t v, uint32_t dv, uint32_t u, uint32_t du) {
  return dv > du || (dv == du && v < u);
}

// The long rows' pieces in tile t: slot 2t, the row u that has the tile's first entry, and slot
// 2t + 1, the row that begins inside the tile and has the next one's first entry (a long row
// is longer than two tiles, so there are no others).  Keepers of every piece into kept[slot],
// the pieces into a list.
__device__ __forceinline__ void dg_count_pieces(const uint32_t *__restrict__ off, const uint32_t *__restrict__ tilerow,
                                                const int32_t *__restrict__ dst, uint32_t m,
                                                uint2 *__restrict__ pieces, uint32_t *__restrict__ kept,
                                                unsigned long long *__restrict__ ctr) {
  static_assert(DG_TILE % 256 == 0, "tiles of the row index");
  __shared__ uint2 s_piece[2 * DG_THREADS];
  __shared__ uint32_t s_pieces, s_sum;
  const uint32_t tiles = m / DG_TILE + (m % DG_TILE ? 1u : 0u);
  // neighbouring tiles to different CTAs
  for (uint32_t t0 = 0; t0 < tiles; t0 += gridDim.x * DG_THREADS) {
    __syncthreads();
    if (threadIdx.x == 0) s_pieces = 0;
    __syncthreads();
    const uint32_t t = t0 + threadIdx.x * gridDim.x + blockIdx.x;
    if (t < tiles) {
      const uint32_t u = __ldg(tilerow + t * (DG_TILE / 256u));
      if (__ldg(off + u + 1) - __ldg(off + u) > 2 * DG_TILE) s_piece[atomicAdd(&s_pieces, 1u)] = make_uint2(u, 2 * t);
      if (t + 1 < tiles) {
        const uint32_t w = __ldg(tilerow + (t + 1) * (DG_TILE / 256u)), b = __ldg(off + w);
        if (w != u && b < (t + 1) * DG_TILE && __ldg(off + w + 1) - b > 2 * DG_TILE)
          s_piece[atomicAdd(&s_pieces, 1u)] = make_uint2(w, 2 * t + 1);
      }
    }
    __syncthreads();
    const uint32_t np = s_pieces;
    for (uint32_t i = 0; i < np; i++) {
      const uint2 pc = s_piece[i];
      const uint32_t u = pc.x, b = __ldg(off + u), end = __ldg(off + u + 1), du = end - b, lo = (pc.y >> 1) * DG_TILE;
      const uint32_t e0 = max(b, lo), len = accx_slice_end(lo, DG_TILE, end) - e0;
      uint32_t c = 0;
      for (uint32_t j0 = threadIdx.x; j0 < len; j0 += 4 * DG_THREADS) {
        uint32_t v[4];
#pragma unroll
        for (int r = 0; r < 4; r++) v[r] = j0 + r * DG_THREADS < len ? (uint32_t)__ldg(dst + e0 + j0 + r * DG_THREADS) : u;
#pragma unroll
        for (int r = 0; r < 4; r++) c += dg_before(v[r], __ldg(off + v[r] + 1) - __ldg(off + v[r]), u, du);
      }
      if (threadIdx.x == 0) s_sum = 0;
      __syncthreads();
      c = __reduce_add_sync(ACCX_FULL_MASK, c);
      if ((threadIdx.x & 31) == 0) atomicAdd(&s_sum, c);
      __syncthreads();
      if (threadIdx.x == 0) {
        kept[pc.y] = s_sum;
        pieces[atomicAdd(&ctr[C_DGLONG], 1ull)] = pc;
      }
    }
  }
}

// F(u) into f[off[u] ..], the entries they came from into ent, their counters zeroed:
// eight lanes a row, 32 entries a step.  Longer rows go to a list.
__global__ void __launch_bounds__(DG_THREADS) k_dg_rows(const uint32_t *__restrict__ off,
                                                        const uint32_t *__restrict__ tilerow,
                                                        const int32_t *__restrict__ dst, uint32_t n, uint32_t m,
                                                        int32_t *__restrict__ f, uint32_t *__restrict__ ent,
                                                        int32_t *__restrict__ fc, uint32_t *__restrict__ flen,
                                                        uint32_t *__restrict__ big, uint32_t *__restrict__ mid,
                                                        uint32_t row, uint2 *__restrict__ pieces,
                                                        uint32_t *__restrict__ kept, unsigned long long *__restrict__ ctr) {
  static_assert(DG_ROW <= DG_WARP, "a listed row's F fits a warp's table");
  // the CTA's rows for the list, placed by one atomic at the end
  __shared__ unsigned long long s_st[9], s_at;
  __shared__ uint32_t s_list[DG_KEEP], s_cnt;
  const int lane = threadIdx.x & 31, gl = lane & 7;
  if (threadIdx.x == 0) s_cnt = 0;
  __syncthreads();
  dg_count_pieces(off, tilerow, dst, m, pieces, kept, ctr);
  const unsigned gmask = 0xffu << (lane & 24);
  cl_stats st;
  const uint32_t ng = gridDim.x * (DG_THREADS / 8);
  for (uint32_t u = blockIdx.x * (DG_THREADS / 8) + threadIdx.x / 8; u < n; u += ng) {
    const uint32_t b = __ldg(off + u), du = __ldg(off + u + 1) - b;
    if (du > row) {
      if (gl == 0 && du <= 2 * DG_TILE) big[atomicAdd(&ctr[C_DGBIG], 1ull)] = u;
      continue;
    }
    uint32_t k = 0;
    for (uint32_t i0 = 0; i0 < du; i0 += 32) {
      uint32_t v[4], dv[4];
#pragma unroll
      for (int r = 0; r < 4; r++) v[r] = i0 + r * 8 + gl < du ? (uint32_t)__ldg(dst + b + i0 + r * 8 + gl) : 0u;
#pragma unroll
      for (int r = 0; r < 4; r++) dv[r] = __ldg(off + v[r] + 1) - __ldg(off + v[r]);
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const bool keep = i0 + r * 8 + gl < du && dg_before(v[r], dv[r], u, du);
        const unsigned bal = (__ballot_sync(gmask, keep) & gmask) >> (lane & 24);
        if (keep) {
          const uint32_t p = b + k + __popc(bal & ((1u << gl) - 1u));
          f[p] = (int32_t)v[r];
          ent[p] = b + i0 + r * 8 + gl;
          fc[p] = 0;
          dg_stat(st, dv[r], du);
        }
        k += __popc(bal);
      }
    }
    if (gl == 0) {
      flen[u] = k;
      if (k > DG_LIGHT) {
        const uint32_t p = atomicAdd(&s_cnt, 1u);
        if (p < DG_KEEP) s_list[p] = u;
        else mid[atomicAdd(&ctr[C_LIGHT], 1ull)] = u;
      }
    }
  }
  dg_stat_flush(st, s_st, ctr);  // its barriers come after the last row
  const uint32_t rows = min(s_cnt, DG_KEEP);
  if (threadIdx.x == 0 && rows) s_at = atomicAdd(&ctr[C_LIGHT], (unsigned long long)rows);
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < rows; i += DG_THREADS) mid[s_at + i] = s_list[i];
}

// The same for the listed rows, a CTA a row or a piece of a long one.
__global__ void __launch_bounds__(DG_THREADS) k_dg_big(const uint32_t *__restrict__ off, const int32_t *__restrict__ dst,
                                                       int32_t *__restrict__ f, uint32_t *__restrict__ ent,
                                                       int32_t *__restrict__ fc, uint32_t *__restrict__ flen,
                                                       const uint32_t *__restrict__ big,
                                                       const uint2 *__restrict__ pieces,
                                                       const uint32_t *__restrict__ kept, uint2 *__restrict__ heavy,
                                                       unsigned long long *__restrict__ ctr) {
  __shared__ unsigned long long s_st[9], s_at;
  __shared__ uint32_t s_w[DG_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  cl_stats st;
  const uint32_t np = (uint32_t)ctr[C_DGLONG], nb = (uint32_t)ctr[C_DGBIG];
  for (uint32_t q = blockIdx.x; q < np + nb; q += gridDim.x) {
    const uint2 pc = q < np ? pieces[q] : make_uint2(big[q - np], 0u);
    const uint32_t u = pc.x, b = __ldg(off + u), end = __ldg(off + u + 1), du = end - b;
    uint32_t e0 = b, e1 = end, k = 0;
    if (q < np) {
      const uint32_t lo = (pc.y >> 1) * DG_TILE, t = b / DG_TILE, pr = (pc.y >> 1) - t;  // pr earlier pieces
      e0 = max(b, lo);
      e1 = accx_slice_end(lo, DG_TILE, end);
      for (uint32_t j = threadIdx.x; j < pr; j += DG_THREADS) k += kept[2 * (t + j) + (j == 0 && b % DG_TILE ? 1 : 0)];
      k = __reduce_add_sync(ACCX_FULL_MASK, k);
      if (lane == 0) s_w[warp] = k;
      __syncthreads();
      k = 0;
      for (int w = 0; w < DG_THREADS / 32; w++) k += s_w[w];
      __syncthreads();
    }
    const uint32_t len = e1 - e0;
    for (uint32_t i0 = 0; i0 < len; i0 += DG_THREADS * 4) {
      uint32_t v[4], dv[4], mine = 0;  // a thread's entries are consecutive: ranks stay in order
      const uint32_t i = i0 + threadIdx.x * 4;
#pragma unroll
      for (int r = 0; r < 4; r++) v[r] = i + r < len ? (uint32_t)__ldg(dst + e0 + i + r) : 0u;
#pragma unroll
      for (int r = 0; r < 4; r++) {
        dv[r] = __ldg(off + v[r] + 1) - __ldg(off + v[r]);
        if (i + r < len && dg_before(v[r], dv[r], u, du)) mine |= 1u << r;
      }
      const uint32_t c = __popc(mine), incl = accx_warp_incl_sum(c, lane);
      if (lane == 31) s_w[warp] = incl;
      __syncthreads();
      uint32_t p = b + k + incl - c;
      for (int w = 0; w < DG_THREADS / 32; w++) {
        if (w < warp) p += s_w[w];
        k += s_w[w];
      }
      for (int r = 0; r < 4; r++)
        if ((mine >> r) & 1u) {
          f[p] = (int32_t)v[r];
          ent[p] = e0 + i + r;
          fc[p] = 0;
          p++;
          dg_stat(st, dv[r], du);
        }
      __syncthreads();
    }
    if (e1 == end) {  // the row's last piece: k is all of F now
      const uint32_t ns = k > 1 ? (du + DG_SLICE - 1) / DG_SLICE : 0u;
      if (threadIdx.x == 0) {
        flen[u] = k;
        if (ns) s_at = atomicAdd(&ctr[C_HEAVY], (unsigned long long)ns);
      }
      __syncthreads();
      for (uint32_t j = threadIdx.x; j < ns; j += DG_THREADS) heavy[s_at + j] = make_uint2(u, j);
      __syncthreads();
    }
  }
  dg_stat_flush(st, s_st, ctr);
}

// One 32-entry step of a row's walk: the lists F(y) of the lanes' y (begin sst, length
// len, 0: none).  Long lists are walked by the whole warp, 128 ids a step; the others
// are concatenated and streamed 32 ids a step, four steps' loads in flight.  lookup(id)
// gives the id's position in the staged F(x) or 0xffffffff.  A hit credits the partner's
// counter fc[j], the owner's oc[position], and the lane's edge.
template <typename L>
__device__ __forceinline__ uint32_t dg_stream(const int32_t *__restrict__ f, int32_t *__restrict__ fc, uint32_t sst,
                                              uint32_t len, or_seg &S, uint32_t *oc, int lane, L lookup) {
  uint32_t hits = 0;
  for (unsigned lm = __ballot_sync(ACCX_FULL_MASK, len >= LONG_SEG); lm; lm &= lm - 1) {
    const int src = __ffs(lm) - 1;
    const uint32_t a0 = __shfl_sync(ACCX_FULL_MASK, sst, src), ln = __shfl_sync(ACCX_FULL_MASK, len, src);
    uint32_t h = 0;
    for (uint32_t i0 = 0; i0 < ln; i0 += 128) {
      int32_t xs[4];
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const uint32_t i = i0 + 32u * r + (uint32_t)lane;
        xs[r] = i < ln ? __ldg(f + a0 + i) : -1;
      }
#pragma unroll
      for (int r = 0; r < 4; r++) {
        if (i0 + 32u * r >= ln) break;
        if (xs[r] < 0) continue;
        const uint32_t p = lookup((uint32_t)xs[r]);
        if (p != 0xffffffffu) {
          atomicAdd(fc + a0 + i0 + 32u * r + (uint32_t)lane, 1);
          atomicAdd(&oc[p], 1u);
          h++;
        }
      }
    }
    h = __reduce_add_sync(ACCX_FULL_MASK, h);
    if (lane == src) hits = h;
  }
  if (len >= LONG_SEG) len = 0;
  const unsigned act = __ballot_sync(ACCX_FULL_MASK, len > 0);
  if (!act) return hits;
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
      const uint32_t i0 = c0 + 32u * r, i = i0 + (uint32_t)lane;
      const uint32_t kb = segb + 1u + (uint32_t)lane;
      const uint32_t o = (kb <= nseg ? S.pre[kb] : 0xffffffffu) - i0;
      const unsigned M = __reduce_or_sync(ACCX_FULL_MASK, o < 32u ? (1u << o) : 0u);
      const uint32_t sj = min(segb + __popc(M & (0xffffffffu >> (31 - lane))), 31u);
      sg[r] = sj;
      gi[r] = (i < tot) ? S.beg[sj] + (i - S.pre[sj]) : 0u;
      xs[r] = (i < tot) ? __ldg(f + gi[r]) : -1;
      segb += __popc(M) + (__ballot_sync(ACCX_FULL_MASK, o == 32u) ? 1u : 0u);
    }
#pragma unroll
    for (int r = 0; r < PROBE_UNROLL; r++) {
      if (xs[r] < 0) continue;
      const uint32_t p = lookup((uint32_t)xs[r]);
      if (p != 0xffffffffu) {
        atomicAdd(fc + gi[r], 1);
        atomicAdd(&oc[p], 1u);
        atomicAdd(&S.hit[sg[r]], 1u);
      }
    }
  }
  __syncwarp();
  if (len) hits = S.hit[me];
  __syncwarp();
  return hits;
}

// The partner list of entry e of row x (|F(x)| = px): begin and length, length 0 where the
// neighbour owns the edge or the row has no such entry.  A neighbour's list is streamed
// when x owns the edge by the longer F (ties: smaller id).
__device__ __forceinline__ uint32_t dg_partner(const uint32_t *__restrict__ off, const int32_t *__restrict__ dst,
                                               const uint32_t *__restrict__ flen, uint32_t x, uint32_t px, uint32_t e,
                                               uint32_t ee, uint32_t *v, uint32_t *sst) {
  *v = 0;
  *sst = 0;
  if (e >= ee) return 0;
  *v = (uint32_t)__ldg(dst + e);
  const uint32_t pv = __ldg(flen + *v);
  if (!accx_owns(x, px, *v, pv)) return 0;
  *sst = __ldg(off + *v);
  return pv;
}

// A row with 2..DG_TINY ids in F and at most DG_TINY_ROW entries, by one lane: the ids in
// registers, four entries' lists in flight.  Partner lists are no longer than its own.  A warp
// a row took 0.6 us of it for two ids: a lattice of 6M vertices 5.2 ms (3.5 by an
// intersection per edge), now 1.3.
__device__ __forceinline__ void dg_tiny_row(const uint32_t *__restrict__ off, const int32_t *__restrict__ dst,
                                            const int32_t *__restrict__ f, const uint32_t *__restrict__ flen, uint32_t x,
                                            uint32_t px, uint32_t b, uint32_t ee, int32_t *__restrict__ fc) {
  int32_t y[DG_TINY];
  uint32_t c[DG_TINY];
#pragma unroll
  for (uint32_t i = 0; i < DG_TINY; i++) {
    y[i] = i < px ? __ldg(f + b + i) : -1;
    c[i] = 0;
  }
  for (uint32_t e0 = b; e0 < ee; e0 += 4) {
    uint32_t v[4], sst[4], len[4];
    int32_t id[4][DG_TINY];
#pragma unroll
    for (int r = 0; r < 4; r++) len[r] = dg_partner(off, dst, flen, x, px, e0 + r, ee, &v[r], &sst[r]);
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
      for (uint32_t j = 0; j < DG_TINY; j++) id[r][j] = j < len[r] ? __ldg(f + sst[r] + j) : -2;
#pragma unroll
    for (int r = 0; r < 4; r++) {
      uint32_t h = 0;
#pragma unroll
      for (uint32_t j = 0; j < DG_TINY; j++) {
        bool hit = false;
#pragma unroll
        for (uint32_t i = 0; i < DG_TINY; i++) {
          const bool q = id[r][j] == y[i];
          c[i] += q;
          hit |= q;
        }
        if (hit) atomicAdd(fc + sst[r] + j, 1);
        h += hit;
      }
      if (!h) continue;
      // the edge's own credit: at the neighbour's place in F(x), or x's in F(v)
      bool here = false;
#pragma unroll
      for (uint32_t i = 0; i < DG_TINY; i++) {
        const bool q = y[i] == (int32_t)v[r];
        c[i] += q ? h : 0u;
        here |= q;
      }
#pragma unroll
      for (uint32_t j = 0; j < DG_TINY; j++)
        if (!here && id[r][j] == (int32_t)x) atomicAdd(fc + sst[r] + j, (int32_t)h);
    }
  }
#pragma unroll
  for (uint32_t i = 0; i < DG_TINY; i++)
    if (c[i]) atomicAdd(fc + b + i, (int32_t)c[i]);
}

// The shorter rows with 2..CAP ids in F, a warp each: F(x) in a hash table of
// ids, with their positions beside it, the row's entries 32 at a time.  (Words of id and
// position took the same time, but only ids of 24 bits.)  CAP = DG_LIGHT: every row, a
// warp's rows spread over the graph (ids near each other often have like degrees); CAP =
// DG_WARP: the listed rows, from a counter.
#define DG_WARPS (DG_THREADS / 32)
template <uint32_t CAP>
struct dg_warp {
  uint32_t tab[4 * CAP];
  uint8_t pos[4 * CAP];
  uint32_t oc[CAP];
  or_seg seg;
};
template <uint32_t CAP>
__global__ void __launch_bounds__(DG_THREADS) k_dg_warp(const uint32_t *__restrict__ off, const int32_t *__restrict__ dst,
                                                        const int32_t *__restrict__ f,
                                                        const uint32_t *__restrict__ flen, uint32_t n,
                                                        const uint32_t *__restrict__ mid, int32_t *__restrict__ fc,
                                                        uint32_t maxrow, unsigned long long *__restrict__ ctr) {
  extern __shared__ __align__(16) uint32_t smem[];
  const int lane = threadIdx.x & 31;
  dg_warp<CAP> &S = reinterpret_cast<dg_warp<CAP> *>(smem)[threadIdx.x >> 5];
  const uint32_t nw = gridDim.x * DG_WARPS, w0 = blockIdx.x * DG_WARPS + (threadIdx.x >> 5);
  auto row = [&](uint32_t x, uint32_t px) {
    const uint32_t b = __ldg(off + x), ee = __ldg(off + x + 1);
    if (CAP == DG_LIGHT && ee - b > maxrow) return;  // walked by CTAs
    int lg = 6;
    while (lg < 10 && (1u << lg) < 4u * px) lg++;
    const uint32_t mask = (1u << lg) - 1u;
    const int sh = 32 - lg;
    for (uint32_t i = lane; i <= mask; i += 32) S.tab[i] = 0xffffffffu;
    for (uint32_t i = lane; i < px; i += 32) S.oc[i] = 0;
    __syncwarp();
    for (uint32_t i = lane; i < px; i += 32) {
      const uint32_t y = (uint32_t)__ldg(f + b + i);
      uint32_t h = ow_hash(y, sh);
      while (atomicCAS(&S.tab[h], 0xffffffffu, y) != 0xffffffffu) h = (h + 1) & mask;
      S.pos[h] = (uint8_t)i;
    }
    __syncwarp();
    auto look = [&](uint32_t id) {
      uint32_t h = ow_hash(id, sh), t = S.tab[h];
      while (t != id && t != 0xffffffffu) {
        h = (h + 1) & mask;
        t = S.tab[h];
      }
      return t == 0xffffffffu ? t : (uint32_t)S.pos[h];
    };
    for (uint32_t e0 = b; e0 < ee; e0 += 32) {
      uint32_t v, sst;
      const uint32_t len = dg_partner(off, dst, flen, x, px, e0 + lane, ee, &v, &sst);
      const uint32_t h = dg_stream(f, fc, sst, len, S.seg, S.oc, lane, look);
      if (h) {  // the edge's own credit: at the neighbour's place in F(x), or x's in F(v)
        const uint32_t p = look(v);
        if (p != 0xffffffffu) atomicAdd(&S.oc[p], h);
        else atomicAdd(fc + accx_lower_bound(f, sst, sst + len, (int32_t)x), (int32_t)h);
      }
    }
    __syncwarp();
    for (uint32_t i = lane; i < px; i += 32) {
      const uint32_t h = S.oc[i];
      if (h) atomicAdd(fc + b + i, (int32_t)h);
    }
    __syncwarp();
  };
  if (CAP == DG_LIGHT) {
    for (unsigned long long x0 = w0; x0 < n; x0 += 32ull * nw) {
      const unsigned long long xl = x0 + (unsigned long long)lane * nw;
      const uint32_t fl = xl < n ? __ldg(flen + xl) : 0u;
      // a single id closes no triangle from here
      bool tiny = fl > 1 && fl <= DG_TINY;
      if (tiny) {
        const uint32_t x = (uint32_t)xl, b = __ldg(off + x), ee = __ldg(off + x + 1);
        tiny = ee - b <= DG_TINY_ROW;
        if (tiny) dg_tiny_row(off, dst, f, flen, x, fl, b, ee, fc);
      }
      __syncwarp();
      for (unsigned rows = __ballot_sync(ACCX_FULL_MASK, fl > 1 && fl <= CAP && !tiny); rows; rows &= rows - 1) {
        const int q = __ffs(rows) - 1;
        row((uint32_t)(x0 + (unsigned long long)q * nw), __shfl_sync(ACCX_FULL_MASK, fl, q));
      }
    }
  } else {
    const uint32_t total = (uint32_t)ctr[C_LIGHT];
    for (;;) {
      uint32_t it = 0;
      if (lane == 0) it = (uint32_t)atomicAdd(&ctr[C_TICKET], 1ull);
      it = __shfl_sync(ACCX_FULL_MASK, it, 0);
      if (it >= total) break;
      const uint32_t x = __ldg(mid + it);
      row(x, __ldg(flen + x));
    }
  }
}

// The listed slices of rows with a longer F or more entries: a CTA each, F staged up to
// DG_CAP ids at a time in a table of ids and positions; warps take 32 entries at a time.
__global__ void __launch_bounds__(DG_THREADS) k_dg_cta(const uint32_t *__restrict__ off, const int32_t *__restrict__ dst,
                                                       const int32_t *__restrict__ f,
                                                       const uint32_t *__restrict__ flen,
                                                       const uint2 *__restrict__ heavy, int32_t *__restrict__ fc,
                                                       unsigned long long *__restrict__ ctr) {
  extern __shared__ __align__(16) uint32_t smem[];
  uint32_t *tab = smem;                                               // DG_SLOTS ids
  uint32_t *oc = tab + DG_SLOTS;                                      // DG_CAP counters
  uint16_t *pos = reinterpret_cast<uint16_t *>(oc + DG_CAP);          // DG_SLOTS positions
  __shared__ or_seg s_seg[DG_WARPS];
  __shared__ uint32_t s_q, s_next;
  const int tid = threadIdx.x, lane = tid & 31;
  or_seg &S = s_seg[tid >> 5];
  const uint32_t nh = (uint32_t)ctr[C_HEAVY];
  for (;;) {
    if (tid == 0) s_q = (uint32_t)atomicAdd(&ctr[C_ITEMS], 1ull);
    __syncthreads();
    if (s_q >= nh) break;
    const uint2 item = heavy[s_q];
    const uint32_t x = item.x, b = __ldg(off + x), px = __ldg(flen + x);
    const uint32_t e0 = b + item.y * DG_SLICE, ee = accx_slice_end(e0, DG_SLICE, __ldg(off + x + 1));
    for (uint32_t c0 = 0; c0 < px; c0 += DG_CAP) {
      const uint32_t cn = min(px - c0, DG_CAP);
      int lg = 8;
      while ((1u << lg) < 4u * cn && (1u << lg) < DG_SLOTS) lg++;
      const uint32_t mask = (1u << lg) - 1u;
      const int sh = 32 - lg;
      for (uint32_t i = tid; i <= mask; i += DG_THREADS) tab[i] = 0xffffffffu;
      for (uint32_t i = tid; i < cn; i += DG_THREADS) oc[i] = 0;
      if (tid == 0) s_next = 0;
      __syncthreads();
      for (uint32_t i = tid; i < cn; i += DG_THREADS) {
        const uint32_t id = (uint32_t)__ldg(f + b + c0 + i);
        uint32_t h = ow_hash(id, sh);
        while (atomicCAS(&tab[h], 0xffffffffu, id) != 0xffffffffu) h = (h + 1) & mask;
        pos[h] = (uint16_t)i;
      }
      __syncthreads();
      auto look = [&](uint32_t id) {
        uint32_t h = ow_hash(id, sh), t = tab[h];
        while (t != id && t != 0xffffffffu) {
          h = (h + 1) & mask;
          t = tab[h];
        }
        return t == 0xffffffffu ? t : (uint32_t)pos[h];
      };
      for (;;) {
        uint32_t e = 0;
        if (lane == 0) e = atomicAdd(&s_next, 32u);
        e = __shfl_sync(ACCX_FULL_MASK, e, 0);
        if (e >= ee - e0) break;
        e += e0;
        uint32_t v, sst;
        const uint32_t len = dg_partner(off, dst, flen, x, px, e + lane, ee, &v, &sst);
        const uint32_t h = dg_stream(f, fc, sst, len, S, oc, lane, look);
        if (h) {  // the edge's own credit: at the neighbour's place in F(x), or x's in F(v)
          const uint32_t p = look(v);
          if (p != 0xffffffffu) {
            atomicAdd(&oc[p], h);
          } else {
            uint32_t lb = b, le = b + px;  // in another part of F(x)?
            if (px > DG_CAP) lb = accx_lower_bound(f, lb, le, (int32_t)v);
            if (px > DG_CAP && lb < le && __ldg(f + lb) == (int32_t)v) atomicAdd(fc + lb, (int32_t)h);
            else atomicAdd(fc + accx_lower_bound(f, sst, sst + len, (int32_t)x), (int32_t)h);
          }
        }
      }
      __syncthreads();
      for (uint32_t i = tid; i < cn; i += DG_THREADS) {
        const uint32_t h = oc[i];
        if (h) atomicAdd(fc + b + c0 + i, (int32_t)h);
      }
      __syncthreads();
    }
  }
}

// Every edge's count, from its place in F to both of its entries.
template <int TILE>
__global__ void __launch_bounds__(TILE) k_dg_out(const uint32_t *__restrict__ off, const uint32_t *__restrict__ tilerow,
                                                 const int32_t *__restrict__ dst, uint32_t n, uint32_t m, int32_t bias,
                                                 const int32_t *__restrict__ f, const uint32_t *__restrict__ ent,
                                                 const int32_t *__restrict__ fc, const uint32_t *__restrict__ flen,
                                                 int32_t *__restrict__ cnt) {
  __shared__ accx_tile_rows<TILE> sh;
  const uint32_t base = blockIdx.x * (uint32_t)TILE, j = base + threadIdx.x;
  const uint32_t u = accx_tile_row<TILE>(off, tilerow, n, m, base, j, &sh);
  if (j >= m || j - __ldg(off + u) >= __ldg(flen + u)) return;
  const int32_t c = fc[j] + bias;
  const uint32_t v = (uint32_t)f[j];
  cnt[ent[j]] = c;
  const uint32_t ve = __ldg(off + v + 1), r = accx_lower_bound(dst, __ldg(off + v), ve, (int32_t)u);
  if (r < ve && __ldg(dst + r) == (int32_t)u) cnt[r] = c;
}

// A small graph in one kernel: a CTA takes DS_TILE entries, keeps the owned ones, and
// gives a warp to each: its lanes search the shorter list's ids in the longer list, and
// the count goes to both entries.  An R-MAT 10 count is launches and little else: nine
// kernels and two fills took 61 us, with the caller's copy; now 18.  Few entries a CTA and
// whole warps, because the hub's row would otherwise be the tail (64 entries and eight
// lanes an edge: 41 us for this kernel alone).  A CTA a tile, but with a limit on the SMs
// only as many CTAs as fit them at once (eight an SM), which loop.
#define DS_TILE 16
__global__ void __launch_bounds__(256) k_count_small(const uint32_t *__restrict__ off,
                                                     const uint32_t *__restrict__ tilerow,
                                                     const int32_t *__restrict__ dst, uint32_t n, uint32_t m,
                                                     int32_t bias, int32_t *cnt, int32_t *copy,
                                                     unsigned long long *__restrict__ ctr) {
  __shared__ unsigned long long s_st[9];
  __shared__ uint4 s_own[DS_TILE];
  __shared__ uint2 s_list[DS_TILE];
  __shared__ uint32_t s_n;
  const int lane = threadIdx.x & 31;
  const uint32_t tiles = (m + DS_TILE - 1) / DS_TILE;
  cl_stats st;
  for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const uint32_t e = tile * DS_TILE + threadIdx.x;
    __syncthreads();  // the list is the last tile's no more
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
    if (threadIdx.x < DS_TILE && e < m) {
      const uint32_t t = e / 256u;
      const uint32_t v = (uint32_t)__ldg(dst + e);
      const uint32_t u = accx_row_of(off, __ldg(tilerow + t), __ldg(tilerow + t + 1) + 1, e);
      const uint32_t ab = __ldg(off + u), ae = __ldg(off + u + 1), vb = __ldg(off + v), ve = __ldg(off + v + 1);
      if (accx_owns(u, ae - ab, v, ve - vb)) {
        const uint32_t i = atomicAdd(&s_n, 1u);
        s_own[i] = make_uint4(ab, ae, vb, ve);
        s_list[i] = make_uint2(u, e);
        dg_stat(st, ae - ab, ve - vb);
      }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x / 32; i < s_n; i += 8) {
      const uint4 o = s_own[i];
      uint32_t lo = o.x, c = 0, r = 0;
      if (lane == 31) r = accx_lower_bound(dst, o.z, o.w, (int32_t)s_list[i].x);  // the reverse entry
      for (uint32_t j0 = o.z; j0 < o.w && lo < o.y; j0 += 32) {
        const uint32_t j = j0 + lane;
        uint32_t p = o.y;
        if (j < o.w) {
          const int32_t id = __ldg(dst + j);
          p = accx_lower_bound(dst, lo, o.y, id);
          c += p < o.y && __ldg(dst + p) == id;
        }
        lo = __shfl_sync(ACCX_FULL_MASK, p, (int)min(o.w - j0 - 1u, 31u));
      }
      c = __reduce_add_sync(ACCX_FULL_MASK, c);
      // lane 0: the entry, lane 31: its reverse
      if (lane == 0) r = s_list[i].y;
      if (lane == 0 || (lane == 31 && r < o.w && __ldg(dst + r) == (int32_t)s_list[i].x)) {
        cnt[r] = (int32_t)c + bias;
        if (copy) copy[r] = (int32_t)c + bias;
      }
    }
  }
  dg_stat_flush(st, s_st, ctr);
}
