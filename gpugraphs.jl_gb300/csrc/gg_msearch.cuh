// gg_msearch.cuh -- device code shared by the batched searches (gg_batch.cu) and
// the query server (gg_serve.cu): many BFS / shortest-path sources advanced together
// over one graph.
//  * BFS: the sources' frontier / visited sets are bits of W <= 8 words per vertex.
//    A level (k_ms_level) ORs the frontier words of a vertex's in-neighbours (edges
//    with odd / true values, the levels semiring of src/algorithms/bfs.jl:52-59) into
//    its unvisited bits, for the sources in `act` only (those whose frontier is not
//    empty); a vertex stops scanning once all of them reached it.  Vertices with more
//    than kCoopDeg in-edges are scanned by the whole warp; hubs (more than kHubDegB)
//    in pieces by separate warps (k_ms_hub), finished by k_ms_hub_final.  New levels
//    are written through an output policy (a distance matrix, or per-query buffers).
//  * Shortest paths: 32 source columns, lane = column, distances vertex-major so one
//    in-neighbour costs one 128-byte read.  A round (k_ms_round) pulls from the
//    in-neighbours whose distances changed in the previous round and lowers D in
//    place; hubs are relaxed in pieces with atomic min (k_ms_round_hub).  The fixpoint
//    is that of shortest_path's Jacobi rounds (src/algorithms/shortest_path.jl:61-80).
#pragma once

#include "gg_queue.cuh"
#include "gg_semiring.cuh"

namespace gg {

int graph_view(gg_ctx* ctx, gg_mat* A, const int32_t** rp, const int32_t** cv, const void** nz,
               bool* all_odd, bool* nonneg);  // gg_graph.cu
int build_hub_plan(gg_ctx* ctx, gg_mat* A, const int32_t* rowptr, int64_t n);  // gg_batch.cu
int push_view(gg_ctx* ctx, gg_mat* A, const int32_t** prow, const int32_t** pcol);  // gg_graph.cu
int sssp_prepare(gg_ctx* ctx, gg_mat* A);  // gg_graph.cu
int weight_sorted_rows(gg_ctx* ctx, gg_mat* A, const int32_t** col, const void** w,
                       double* mean_w);  // gg_graph.cu

namespace {

static const unsigned kFullB = 0xffffffffu;
static const int kMaxW = 8;  // 256 sources per BFS group

struct BatchGraph {  // CSR view of A_T used by the batched kernels
  const int32_t* rowptr;
  const int32_t* colval;
  const void* nz;
  int tv;
  bool odd_only;
};

__device__ __forceinline__ bool b_odd(const void* nz, int tv, int64_t k) {
  switch (tv) {
    case GG_BOOL: return static_cast<const uint8_t*>(nz)[k] & 1;
    case GG_INT32: return static_cast<const int32_t*>(nz)[k] & 1;
    case GG_INT64: return static_cast<const int64_t*>(nz)[k] & 1;
  }
  return false;
}

static const int kCoopDeg = 32;  // in-degree above which the whole warp scans a vertex

// output policies of the BFS kernels: source column q reached vertex v this level
struct LevelOutMatrix {  // dist[q * ld + v] = level
  int32_t* dist;
  int64_t ld;
  int32_t level;
  __device__ __forceinline__ void put(int q, int64_t v) const { dist[(int64_t)q * ld + v] = level; }
};
struct LevelOutSlots {  // per-query buffers: out[q][v] = tick - start[q]
  int32_t* const* outp;
  const int32_t* start;
  int32_t tick;
  __device__ __forceinline__ void put(int q, int64_t v) const { outp[q][v] = tick - start[q]; }
};

// OR of the frontier words of in-edges [k0, k1) of one vertex, the whole warp
// scanning 32 edges per step; stops once every bit of m is set.  Uniform result.
template <int W>
__device__ __forceinline__ void warp_scan_or(const BatchGraph& g, const unsigned* __restrict__ F,
                                             int64_t k0, int64_t k1, const unsigned (&m)[W],
                                             unsigned (&acc)[W], int lane) {
#pragma unroll
  for (int w = 0; w < W; ++w) acc[w] = 0;
  for (int64_t kb = k0; kb < k1; kb += 32) {
    const int64_t k = kb + lane;
    unsigned f[W];
#pragma unroll
    for (int w = 0; w < W; ++w) f[w] = 0;
    if (k < k1 && (!g.odd_only || b_odd(g.nz, g.tv, k))) {
      const int64_t u = (int64_t)__ldg(g.colval + k) - 1;
#pragma unroll
      for (int w = 0; w < W; ++w) f[w] = __ldg(F + u * W + w);
    }
    bool full = true;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      acc[w] |= __reduce_or_sync(kFullB, f[w]);
      full &= (acc[w] & m[w]) == m[w];
    }
    if (full) break;
  }
}

// one bottom-up level for a group of sources (W words per vertex); act holds the
// sources whose frontier is non-empty, act_next collects those of the next level
template <int W, class Out>
__global__ void __launch_bounds__(256)
    k_ms_level(int64_t n, BatchGraph g, const unsigned* __restrict__ F, unsigned* Fn,
               unsigned* V, const unsigned* __restrict__ act, unsigned* act_next, Out out,
               unsigned long long* count) {
  const int lane = threadIdx.x & 31;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  unsigned am[W];
#pragma unroll
  for (int w = 0; w < W; ++w) am[w] = act[w];
  for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < n; base += stride) {
    const int64_t v = base + threadIdx.x;
    unsigned m[W], acc[W];
    bool open = false, hub = false;
    int64_t k0 = 0, k1 = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      m[w] = 0;
      acc[w] = 0;
    }
    if (v < n) {
      k0 = (int64_t)g.rowptr[v] - 1;
      k1 = (int64_t)g.rowptr[v + 1] - 1;
      hub = k1 - k0 > kHubDegB;
      if (!hub) {
#pragma unroll
        for (int w = 0; w < W; ++w) {
          m[w] = ~V[v * W + w] & am[w];
          open |= m[w] != 0;
        }
      }
    }
    const bool light = open && k1 - k0 <= kCoopDeg;
    if (light) {
      for (int64_t k = k0; k < k1; ++k) {
        if (g.odd_only && !b_odd(g.nz, g.tv, k)) continue;
        const int64_t u = (int64_t)__ldg(g.colval + k) - 1;
        bool full = true;
#pragma unroll
        for (int w = 0; w < W; ++w) {
          acc[w] |= __ldg(F + u * W + w);
          full &= (acc[w] & m[w]) == m[w];
        }
        if (full) break;  // every open source reached this vertex
      }
    }
    unsigned coop = __ballot_sync(kFullB, open && !light);
    while (coop) {
      const int h = __ffs(coop) - 1;
      coop &= coop - 1;
      unsigned hm[W], ha[W];
#pragma unroll
      for (int w = 0; w < W; ++w) hm[w] = __shfl_sync(kFullB, m[w], h);
      warp_scan_or<W>(g, F, __shfl_sync(kFullB, k0, h), __shfl_sync(kFullB, k1, h), hm, ha, lane);
      if (lane == h) {
#pragma unroll
        for (int w = 0; w < W; ++w) acc[w] = ha[w];
      }
    }
    unsigned anynew = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      acc[w] &= m[w];
      anynew |= acc[w];
      if (v < n && !hub) {  // hubs are finished by k_ms_hub_final
        if (acc[w]) V[v * W + w] |= acc[w];
        Fn[v * W + w] = acc[w];
      }
    }
    // level writes, one source column at a time (coalesced over the warp's vertices)
#pragma unroll
    for (int w = 0; w < W; ++w) {
      const unsigned any_w = __reduce_or_sync(kFullB, acc[w]);
      if (lane == 0 && any_w) atomicOr(act_next + w, any_w);
      unsigned u = any_w;
      while (u) {
        const int b = __ffs(u) - 1;
        u &= u - 1;
        if ((acc[w] >> b) & 1u) out.put(w * 32 + b, v);
      }
    }
    const unsigned bal = __ballot_sync(kFullB, anynew != 0);
    if (lane == 0 && bal) atomicAdd(count, (unsigned long long)__popc(bal));
  }
}

// hub pieces: one warp per piece ORs its in-neighbours' frontier words into the
// hub's accumulator
template <int W>
__global__ void __launch_bounds__(256)
    k_ms_hub(BatchGraph g, const int4* __restrict__ pieces, int64_t npiece,
             const int32_t* __restrict__ hubs, const unsigned* __restrict__ F,
             const unsigned* __restrict__ V, const unsigned* __restrict__ act, unsigned* hacc) {
  const int lane = threadIdx.x & 31;
  for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < npiece;
       i += ((int64_t)gridDim.x * blockDim.x) >> 5) {
    const int4 p = pieces[i];
    const int64_t v = hubs[p.x];
    unsigned m[W], ha[W];
    bool open = false;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      m[w] = ~V[v * W + w] & act[w];
      open |= m[w] != 0;
    }
    if (!open) continue;
    warp_scan_or<W>(g, F, p.y, p.z, m, ha, lane);
    if (lane == 0) {
#pragma unroll
      for (int w = 0; w < W; ++w)
        if (ha[w] & m[w]) atomicOr(hacc + (int64_t)p.x * kMaxW + w, ha[w] & m[w]);
    }
  }
}

// one thread per hub: new bits, visited, next frontier, levels
template <int W, class Out>
__global__ void k_ms_hub_final(const int32_t* __restrict__ hubs, int64_t nhub, unsigned* hacc,
                               unsigned* Fn, unsigned* V, const unsigned* __restrict__ act,
                               unsigned* act_next, Out out, unsigned long long* count) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nhub;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t v = hubs[i];
    bool any = false;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      const unsigned m = ~V[v * W + w] & act[w];
      const unsigned a = hacc[i * kMaxW + w] & m;
      hacc[i * kMaxW + w] = 0;
      Fn[v * W + w] = a;
      if (!a) continue;
      any = true;
      V[v * W + w] |= a;
      atomicOr(act_next + w, a);
      unsigned u = a;
      while (u) {
        const int b = __ffs(u) - 1;
        u &= u - 1;
        out.put(w * 32 + b, v);
      }
    }
    if (any) atomicAdd(count, 1ull);
  }
}

template <typename T> __device__ __forceinline__ T b_relax(T w, T d) {
  return (w == Lim<T>::max() || d == Lim<T>::max()) ? Lim<T>::max() : w_add(w, d);
}

template <typename T>
__device__ __forceinline__ T b_weight(const void* nz, int tv, int64_t k) {
  switch (tv) {
    case GG_BOOL: return static_cast<T>(static_cast<const uint8_t*>(nz)[k]);
    case GG_INT32: return static_cast<T>(static_cast<const int32_t*>(nz)[k]);
    case GG_INT64: return static_cast<T>(static_cast<const int64_t*>(nz)[k]);
    case GG_FLOAT32: return static_cast<T>(static_cast<const float*>(nz)[k]);
  }
  return static_cast<T>(static_cast<const double*>(nz)[k]);
}

// pull over in-edges [k0, k1) of v from in-neighbours that changed last round or
// already in this one: per-lane (source column) minimum of D[u] + w.  chg[u] holds the
// columns of u that dropped in the previous round, chg_cur[u] those dropped so far in
// this round (a drop made earlier in the round travels on at once, so fewer rounds
// are needed; any order of relaxations reaches the same fixpoint); only those lanes
// read D[u], so a vertex whose distances changed for few sources costs few 32-byte
// sectors.
template <typename T>
__device__ __forceinline__ bool bs_pull(const BatchGraph& g, const T* D,
                                        const unsigned* __restrict__ chg, const unsigned* chg_cur,
                                        int64_t k0, int64_t k1, int lane, T& best) {
  bool any = false;
  // columns and masks of 128 edges in flight (few of a late round's neighbours changed: a
  // 2048-edge hub piece was 64 chains of two round trips)
  for (int64_t kb4 = k0; kb4 < k1; kb4 += 128) {
   int32_t c4[4];
   unsigned m4[4];
#pragma unroll
   for (int t = 0; t < 4; ++t)
     c4[t] = kb4 + t * 32 + lane < k1 ? __ldg(g.colval + kb4 + t * 32 + lane) - 1 : -1;
#pragma unroll
   for (int t = 0; t < 4; ++t) m4[t] = c4[t] >= 0 ? (__ldcg(chg + c4[t]) | __ldcg(chg_cur + c4[t])) : 0u;
#pragma unroll
   for (int t4 = 0; t4 < 4; ++t4) {
    const int64_t kk = kb4 + t4 * 32 + lane;
    const unsigned cm = m4[t4];
    const int32_t u = cm ? c4[t4] : -1;
    const T wl = cm ? b_weight<T>(g.nz, g.tv, kk) : T(0);
    unsigned act = __ballot_sync(kFullB, u >= 0);
    // changed in-neighbours 8 at a time: their rows of D are read together, so a warp
    // keeps up to 8 reads in flight (the minimum does not depend on the order)
    while (act) {
      int32_t su[8];
      unsigned sm[8];
      T sw[8], dv[8];
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        const int src_lane = act ? __ffs(act) - 1 : 0;
        const bool valid = act != 0;
        act &= act - 1;
        su[t] = __shfl_sync(kFullB, u, src_lane);
        sm[t] = valid ? __shfl_sync(kFullB, cm, src_lane) : 0u;
        sw[t] = __shfl_sync(kFullB, wl, src_lane);
      }
#pragma unroll
      for (int t = 0; t < 8; ++t)
        dv[t] = ((sm[t] >> lane) & 1u) ? D[(int64_t)su[t] * 32 + lane] : Lim<T>::max();
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        if ((sm[t] >> lane) & 1u) {
          const T cand = b_relax(sw[t], dv[t]);
          if (cand < best) best = cand;
          any = true;
        }
      }
    }
   }
  }
  return any;
}

// Changed-vertex bookkeeping of a round: chg_next[v] gets the columns that dropped and,
// when cq is given, v is appended to the changed queue cq (count *ncq) that drives the
// next round's marking.
__device__ __forceinline__ void ms_changed(int64_t v, unsigned cols, unsigned* chg_next,
                                           unsigned long long* count, int32_t* cq,
                                           unsigned long long* ncq) {
  atomicOr(chg_next + v, cols);
  atomicAdd(count, 1ull);
  if (cq) cq[atomicAdd(ncq, 1ull)] = (int32_t)v;
}

template <typename T> __device__ __forceinline__ unsigned ms_dist_bits(T d) {
  if constexpr (sizeof(T) == 4) return *reinterpret_cast<const unsigned*>(&d);
  return 0u;  // (8-byte distances: not noted)
}

// what a round's kernels found beside the changed vertices: (vertex, column) pairs that
// dropped, and the smallest distance written, kept as ~(its bits) under max so that the
// cleared word means none (4-byte distances, which order as their bits do).  Null
// pointers: not wanted.
struct MsSums {
  unsigned long long* pairs;
  unsigned long long* low;
  template <typename T>
  __device__ __forceinline__ void add(unsigned long long n, T d) const {  // the whole warp
    if (!pairs) return;
    warp_add(n, pairs);
    const unsigned b = __reduce_max_sync(kFullB, ~ms_dist_bits<T>(d));
    if ((threadIdx.x & 31) == 0 && b != ~ms_dist_bits<T>(Lim<T>::max()))
      atomicMax(low, (unsigned long long)b);
  }
};

// one round: warp per vertex v (every vertex, or the marked ones in vlist[0, *nlist)),
// lane = source column; pull from in-neighbours that changed last round, lower D[v]
// in place, flag v when any column dropped (chg_next is cleared before the round).
// Hubs are left to k_ms_round_hub.
template <typename T>
__global__ void __launch_bounds__(256)
    k_ms_round(int64_t n, BatchGraph g, T* D, const unsigned* __restrict__ chg,
               unsigned* chg_next, unsigned long long* count, unsigned* drop,
               const int32_t* __restrict__ vlist, const unsigned long long* nlist, int32_t* cq,
               unsigned long long* ncq, MsSums sums) {
  const int lane = threadIdx.x & 31;
  unsigned dropped_cols = 0;
  unsigned long long pairs = 0;
  T low = Lim<T>::max();
  const int64_t total = vlist ? (int64_t)*((volatile const unsigned long long*)nlist) : n;
  const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  // the warp's vertices gw, gw + nw, ... taken 32 at a time: vertex j of a batch has its
  // id and row bounds loaded by lane j up front, and the batch's changed vertices are
  // counted and queued with one atomic each
  for (int64_t i0 = gw; i0 < total; i0 += 32 * nw) {
    const int64_t ij = i0 + (int64_t)lane * nw;
    int64_t vj = -1, k0j = 0, k1j = 0;
    if (ij < total) {
      vj = vlist ? (int64_t)vlist[ij] : ij;
      k0j = (int64_t)g.rowptr[vj] - 1;
      k1j = (int64_t)g.rowptr[vj + 1] - 1;
    }
    const unsigned live = __ballot_sync(kFullB, vj >= 0);
    unsigned my_cols = 0;  // lane j: the columns that dropped for vertex j
    for (int j = 0; j < 32 && ((live >> j) & 1u); ++j) {
      const int64_t v = __shfl_sync(kFullB, vj, j);
      const int64_t k0 = __shfl_sync(kFullB, k0j, j), k1 = __shfl_sync(kFullB, k1j, j);
      if (k1 - k0 > kHubDegB) continue;
      T best = Lim<T>::max();
      const bool any = bs_pull<T>(g, D, chg, chg_next, k0, k1, lane, best);
      bool dropped = false;
      if (any) {
        T* dv = D + v * 32 + lane;
        if (best < *dv) {
          *dv = best;
          dropped = true;
          low = best < low ? best : low;
          ++pairs;
        }
      }
      const unsigned b = __ballot_sync(kFullB, dropped);
      dropped_cols |= b;
      if (lane == j) my_cols = b;
    }
    if (my_cols) atomicOr(chg_next + vj, my_cols);
    const unsigned cm = __ballot_sync(kFullB, my_cols != 0);
    if (cm) {
      unsigned long long qb = 0;
      if (lane == 0) {
        atomicAdd(count, (unsigned long long)__popc(cm));
        if (cq) qb = atomicAdd(ncq, (unsigned long long)__popc(cm));
      }
      qb = __shfl_sync(kFullB, qb, 0);
      if (cq && my_cols) cq[qb + __popc(cm & ((1u << lane) - 1u))] = (int32_t)vj;
    }
  }
  if (drop && lane == 0 && dropped_cols) atomicOr(drop, dropped_cols);
  sums.add<T>(pairs, low);
}

// marking for a frontier-restricted round: the out-neighbours of the changed vertices
// cq[0, *ncq) are the only vertices whose distances can drop; each is marked once in
// the bitmap and listed in vlist.  A changed vertex with more than kMarkHub out-edges
// is not walked by one warp (a hub's list held one warp for milliseconds while the
// others idled): it is queued in mhq and its out-list marked in pieces of kMarkPiece
// edges by every warp (k_ms_mark_offsets, k_ms_mark_hub).
static const int kMarkHub = 1024, kMarkPiece = 1024;

__device__ __forceinline__ void ms_mark_range(const int32_t* __restrict__ pcol, int32_t k0,
                                              int32_t k1, int lane, unsigned* mark, int32_t* vlist,
                                              unsigned long long* nlist) {
  for (int32_t kb = k0; kb < k1; kb += 32) {
    const int32_t k = kb + lane;
    bool add = false;
    int32_t w = 0;
    if (k < k1) {
      w = __ldg(pcol + k);
      const unsigned bit = 1u << (w & 31);
      if (!(__ldcg(mark + (w >> 5)) & bit)) add = !(atomicOr(mark + (w >> 5), bit) & bit);
    }
    const unsigned b = __ballot_sync(kFullB, add);
    if (b) {
      const int leader = __ffs(b) - 1;
      unsigned long long base = 0;
      if (lane == leader) base = atomicAdd(nlist, (unsigned long long)__popc(b));
      base = __shfl_sync(kFullB, base, leader);
      if (add) vlist[base + __popc(b & ((1u << lane) - 1u))] = w;
    }
  }
}

__global__ void __launch_bounds__(256)
    k_ms_mark(const int32_t* __restrict__ prow, const int32_t* __restrict__ pcol,
              const int32_t* __restrict__ cq, const unsigned long long* ncq, unsigned* mark,
              int32_t* vlist, unsigned long long* nlist, int32_t* mhq, unsigned long long* nmh) {
  const int lane = threadIdx.x & 31;
  const int64_t total = (int64_t)*((volatile const unsigned long long*)ncq);
  for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < total;
       i += ((int64_t)gridDim.x * blockDim.x) >> 5) {
    const int32_t u = cq[i];
    const int32_t k0 = prow[u], k1 = prow[u + 1];
    if (k1 - k0 > kMarkHub) {  // left to the piece kernel
      if (lane == 0) mhq[atomicAdd(nmh, 1ull)] = u;
      continue;
    }
    ms_mark_range(pcol, k0, k1, lane, mark, vlist, nlist);
  }
}

// piece offsets of the queued hubs: mhoff[h] = pieces of hubs before h, mhoff[nh] = all
__global__ void __launch_bounds__(1024)
    k_ms_mark_offsets(const int32_t* __restrict__ prow, const int32_t* __restrict__ mhq,
                      const unsigned long long* nmh, int32_t* mhoff) {
  __shared__ int32_t wsum[32];
  __shared__ int32_t carry;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t nh = (int64_t)*((volatile const unsigned long long*)nmh);
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int64_t b0 = 0; b0 < nh; b0 += 1024) {
    const int64_t i = b0 + threadIdx.x;
    int32_t np = 0;
    if (i < nh) {
      const int32_t u = mhq[i];
      np = (prow[u + 1] - prow[u] + kMarkPiece - 1) / kMarkPiece;
    }
    int32_t x = np;  // inclusive scan within the warp, then over the warp totals
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t t = __shfl_up_sync(kFullB, x, o);
      if (lane >= o) x += t;
    }
    if (lane == 31) wsum[wid] = x;
    __syncthreads();
    if (wid == 0) {
      int32_t y = wsum[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int32_t t = __shfl_up_sync(kFullB, y, o);
        if (lane >= o) y += t;
      }
      wsum[lane] = y;
    }
    __syncthreads();
    const int32_t incl = x + (wid > 0 ? wsum[wid - 1] : 0);
    const int32_t c = carry;
    if (i < nh) mhoff[i] = c + incl - np;
    __syncthreads();
    if (threadIdx.x == 1023) carry = c + incl;
    __syncthreads();
  }
  if (threadIdx.x == 0) mhoff[nh] = carry;
}

__global__ void __launch_bounds__(256)
    k_ms_mark_hub(const int32_t* __restrict__ prow, const int32_t* __restrict__ pcol,
                  const int32_t* __restrict__ mhq, const unsigned long long* nmh,
                  const int32_t* __restrict__ mhoff, unsigned* mark, int32_t* vlist,
                  unsigned long long* nlist) {
  const int lane = threadIdx.x & 31;
  const int64_t nh = (int64_t)*((volatile const unsigned long long*)nmh);
  if (nh == 0) return;
  const int64_t npieces = mhoff[nh];
  int64_t h = 0;
  for (int64_t q = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < npieces;
       q += ((int64_t)gridDim.x * blockDim.x) >> 5) {
    // the hub holding piece q (q only grows, so search forward from the last one)
    if (__ldg(mhoff + h + 1) <= q) {
      int64_t lo = h + 1, hi = nh - 1;
      while (lo < hi) {
        const int64_t mid = (lo + hi + 1) >> 1;
        if (__ldg(mhoff + mid) <= q) lo = mid; else hi = mid - 1;
      }
      h = lo;
    }
    const int32_t u = mhq[h];
    const int32_t k0 = prow[u] + (int32_t)(q - mhoff[h]) * kMarkPiece;
    const int32_t k1 = min(prow[u + 1], k0 + kMarkPiece);
    ms_mark_range(pcol, k0, k1, lane, mark, vlist, nlist);
  }
}

// the three marking launches of a frontier-restricted round; nmh: a device counter,
// mhq / mhoff: room for n and n + 1 entries
static inline cudaError_t launch_ms_mark(cudaStream_t st, int num_sms, int64_t nchanged,
                                         const int32_t* prow, const int32_t* pcol,
                                         const int32_t* cq, const unsigned long long* ncq,
                                         unsigned* mark, int32_t* vlist, unsigned long long* nlist,
                                         int32_t* mhq, unsigned long long* nmh, int32_t* mhoff) {
  cudaError_t e = cudaMemsetAsync(nmh, 0, sizeof(unsigned long long), st);
  if (e != cudaSuccess) return e;
  int64_t mb = (nchanged * 32 + 255) / 256;
  const int64_t gcap = (int64_t)num_sms * 8;
  if (mb > gcap) mb = gcap;
  k_ms_mark<<<(int)(mb < 1 ? 1 : mb), 256, 0, st>>>(prow, pcol, cq, ncq, mark, vlist, nlist, mhq, nmh);
  k_ms_mark_offsets<<<1, 1024, 0, st>>>(prow, mhq, nmh, mhoff);
  k_ms_mark_hub<<<(int)gcap, 256, 0, st>>>(prow, pcol, mhq, nmh, mhoff, mark, vlist, nlist);
  return cudaGetLastError();
}

template <typename T> __device__ __forceinline__ T b_atomic_min(T* p, T v);
template <> __device__ __forceinline__ int32_t b_atomic_min<int32_t>(int32_t* p, int32_t v) {
  return atomicMin(p, v);
}
template <> __device__ __forceinline__ int64_t b_atomic_min<int64_t>(int64_t* p, int64_t v) {
  return (int64_t)atomicMin((long long*)p, (long long)v);
}
// distances are non-negative here (never -0.0: +0.0 + w), so floats order like
// their bit patterns
template <> __device__ __forceinline__ float b_atomic_min<float>(float* p, float v) {
  return __int_as_float(atomicMin((int*)p, __float_as_int(v)));
}
template <> __device__ __forceinline__ double b_atomic_min<double>(double* p, double v) {
  return __longlong_as_double(atomicMin((long long*)p, __double_as_longlong(v)));
}

// Round over every row (4-byte distances, rows with their entries by ascending weight):
// 8 lanes take a row of up to kSegMM entries or a piece of a longer one, 4 source columns a
// lane with their minima in registers, four rows of about one length a warp (the SpMM
// plan's lists).  An entry costs a 16-byte load of D and four add-min instructions a
// lane; 4 entries' loads are in flight, the next 8 columns and weights behind them.
//  * A row ends at the first weight w with w + dlow >= the largest of its 32 minima, or
//    w > cap: sums of non-negative values only grow, and no distance below dlow was written
//    in the previous round, so an unchanged or pruned entry cannot lower it.  cap < max
//    leaves heavy entries out altogether; a later round must then visit every row with
//    dlow = 0 and no cap before the result is final.
//  * kCheck: entries whose in-neighbour did not change in the previous round are left out
//    by its column mask (worth its gather once few of the pairs drop).  On thin graphs what
//    has dropped in this round so far counts too, as in bs_pull: a tenth fewer of the many
//    rounds of a grid.
// Whole rows have one writer; pieces lower their row by atomic min.  Any order of
// relaxations reaches the same fixpoint.
// Against the round it replaces (a warp per 32-row SELL item, changed entries through a
// shared-memory queue, 19.5 warp instructions an entry, all entries): 800 -> 250 us on R-MAT
// scale 20, 32 Int32 columns; 256 sources 57.5 -> 25.5 ms.  A round alone takes 260 us:
// issue 55%, 45% of the warp slots, L2 20%, DRAM 18%, most stalls on the rows of D.
static const int64_t kMsThin = 8;
struct MsRows {
  const int32_t* rowptr;  // 1-based
  const int32_t* col;     // 1-based, entries of a row by ascending weight
  const void* w;
  int tv;
  const int4* items;      // rows of more than 32 entries and pieces: (row, first, end, piece or -1)
  int64_t nitems;
  const int32_t* short_rows;  // rows of 1..32 entries
  int64_t nshort;
  bool thin;                  // fewer than kMsThin entries a row in the mean
};

// the row rounds' view of A (CSR handles with 1- or 4-byte values; out->col stays nullptr
// for others and where the sorted rows do not fit) and the mean weight
static inline int ms_rows_of(gg_ctx* ctx, gg_mat* A, MsRows* out, double* mean_w) {
  *out = MsRows{};
  GG_CHECK(weight_sorted_rows(ctx, A, &out->col, &out->w, mean_w));
  if (!out->col) return GG_OK;
  GG_CHECK(build_mm_plan(ctx, A));
  const MMPlan* P = A->mmplan;
  out->rowptr = A->rowptr;
  out->tv = A->dtype;
  out->items = P->items;
  out->nitems = P->nitems;
  out->short_rows = P->short_rows;
  out->nshort = P->nlive;
  out->thin = A->nnz < kMsThin * A->m;
  return GG_OK;
}

template <typename T> __device__ __forceinline__ T ms_unbits(int b);
template <> __device__ __forceinline__ int32_t ms_unbits<int32_t>(int b) { return b; }
template <> __device__ __forceinline__ float ms_unbits<float>(int b) { return __int_as_float(b); }
// min(best, w + d) on non-negative values; a sum past Int32 (an unreached d among them)
// stays above every distance
__device__ __forceinline__ int32_t ms_relax(int32_t best, int32_t w, int32_t d) {
  return (int32_t)__viaddmin_u32((unsigned)w, (unsigned)d, (unsigned)best);
}
__device__ __forceinline__ float ms_relax(float best, float w, float d) {
  return fminf(best, __fadd_rn(w, d));
}

// 4 entries of a row with their D rows in flight and 40 warps an SM: 8 entries with 24 / 32
// warps 35.5 / 33.0 ms, 4 with 32 / 40 / 48 (spills) 32.5 / 31.9 / 37.1 ms (256 sources,
// R-MAT scale 20)
static const int kMsRowStep = 4;
static const int kMsRowBlocks = 5;  // CTAs of 256 threads an SM

template <typename T, bool kCheck>
__global__ void __launch_bounds__(256, kMsRowBlocks)
    k_ms_round_rows(MsRows g, T* D, const unsigned* __restrict__ chg, unsigned* chg_next,
                    unsigned long long* count, unsigned* drop, int32_t* cq, unsigned long long* ncq,
                    MsSums sums, T dlow, T cap) {
  __shared__ int32_t stage[8][WarpQueue::kCap];
  const int lane = threadIdx.x & 31, sub = lane & 7, lead = lane & ~7;
  const unsigned gmask = 0xffu << lead;
  WarpQueue wq(stage[threadIdx.x >> 5], cq, ncq);
  unsigned dropped_cols = 0;
  unsigned long long pairs = 0, changed = 0;
  T low = Lim<T>::max();
  const T far_t = Lim<T>::max();
  const int far = *reinterpret_cast<const int*>(&far_t);
  const int64_t total = g.nitems + g.nshort;
  // warps numbered across the blocks first: the longest rows go to different SMs
  const int64_t gw = (int64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x;
  const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t id0 = gw * 4; id0 < total; id0 += nw * 4) {
    const int64_t id = id0 + (lane >> 3);
    int32_t v = -1, k = 0, k1 = 0;
    bool piece = false;
    if (id < g.nitems) {
      const int4 d = __ldg(g.items + id);
      v = d.x;
      k = d.y;
      k1 = d.z;
      piece = d.w >= 0;
    } else if (id < total) {
      v = __ldg(g.short_rows + (id - g.nitems));
      k = __ldg(g.rowptr + v) - 1;
      k1 = __ldg(g.rowptr + v + 1) - 1;
    }
    int32_t c = k + sub < k1 ? __ldg(g.col + k + sub) : 0;
    T w = k + sub < k1 ? b_weight<T>(g.w, g.tv, k + sub) : Lim<T>::max();
    T* row = D + (int64_t)(v < 0 ? 0 : v) * 32 + sub * 4;
    T cur[4], best[4];
    {
      const int4 r = v >= 0 ? __ldcg(reinterpret_cast<const int4*>(row)) : make_int4(0, 0, 0, 0);
      cur[0] = ms_unbits<T>(r.x);
      cur[1] = ms_unbits<T>(r.y);
      cur[2] = ms_unbits<T>(r.z);
      cur[3] = ms_unbits<T>(r.w);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) best[q] = cur[q];
    for (; __any_sync(kFullB, k < k1); k += 8) {
      // the largest of the row's minima so far, and the entries it still admits
      T top = best[0] > best[1] ? best[0] : best[1];
      const T t2 = best[2] > best[3] ? best[2] : best[3];
      top = t2 > top ? t2 : top;
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) {
        const T t = __shfl_xor_sync(kFullB, top, o);
        top = t > top ? t : top;
      }
      const bool in = c > 0 && b_relax(w, dlow) < top && w <= cap;
      if (!in) c = 0;
      const unsigned any = __ballot_sync(kFullB, in);
      if (!(any & gmask)) k = k1;  // ascending weights: nothing of the row is left
      if (!any) break;
      const int32_t kn = k + 8 + sub;
      const int32_t cn = kn < k1 ? __ldg(g.col + kn) : 0;
      const T wn = kn < k1 ? b_weight<T>(g.w, g.tv, kn) : Lim<T>::max();
      unsigned m = ~0u;
      if (kCheck) {
        m = c > 0 ? __ldg(chg + (c - 1)) : 0u;
        if (g.thin && c > 0) m |= __ldcg(chg_next + (c - 1));
      }
#pragma unroll
      for (int h = 0; h < 8; h += kMsRowStep) {
        int4 dv[kMsRowStep];
#pragma unroll
        for (int u = 0; u < kMsRowStep; ++u) {
          const int32_t cu = __shfl_sync(kFullB, c, lead + h + u);
          bool need = cu > 0;
          if constexpr (kCheck) {
            const unsigned mu = __shfl_sync(kFullB, m, lead + h + u);  // every lane takes part
            need = need && ((mu >> (sub * 4)) & 15u);
          }
          dv[u] = need ? __ldcg(reinterpret_cast<const int4*>(D + (int64_t)(cu - 1) * 32 + sub * 4))
                       : make_int4(far, far, far, far);
        }
#pragma unroll
        for (int u = 0; u < kMsRowStep; ++u) {
          const T wu = __shfl_sync(kFullB, w, lead + h + u);
          best[0] = ms_relax(best[0], wu, ms_unbits<T>(dv[u].x));
          best[1] = ms_relax(best[1], wu, ms_unbits<T>(dv[u].y));
          best[2] = ms_relax(best[2], wu, ms_unbits<T>(dv[u].z));
          best[3] = ms_relax(best[3], wu, ms_unbits<T>(dv[u].w));
        }
      }
      c = cn;
      w = wn;
    }
    unsigned bits = 0;
    if (v >= 0) {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (best[q] < cur[q] && (!piece || best[q] < b_atomic_min<T>(row + q, best[q]))) {
          bits |= 1u << q;
          low = best[q] < low ? best[q] : low;
        }
      if (bits && !piece)
        __stcg(reinterpret_cast<int4*>(row), *reinterpret_cast<const int4*>(best));
      pairs += __popc(bits);
    }
    unsigned cols = bits << (sub * 4);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) cols |= __shfl_xor_sync(kFullB, cols, o);
    dropped_cols |= cols;
    bool fresh = false;  // first to flag the row this round
    if (sub == 0 && cols) {
      if (piece) {
        fresh = atomicOr(chg_next + v, cols) == 0u;
      } else {
        chg_next[v] = cols;
        fresh = true;
      }
    }
    changed += fresh;
    wq.push(fresh, v);
  }
  wq.flush();
  warp_add(changed, count);
  if (drop) {
    dropped_cols = __reduce_or_sync(kFullB, dropped_cols);
    if (lane == 0 && dropped_cols) atomicOr(drop, dropped_cols);
  }
  sums.add<T>(pairs, low);
}

// hub pieces: one warp per piece, atomic min into the hub's 32 columns
// (with mark given, only hubs marked for this round are relaxed)
template <typename T>
__global__ void __launch_bounds__(256)
    k_ms_round_hub(BatchGraph g, const int4* __restrict__ pieces, int64_t npiece,
                   const int32_t* __restrict__ hubs, T* D, const unsigned* __restrict__ chg,
                   unsigned* chg_next, unsigned long long* count, unsigned* drop,
                   const unsigned* __restrict__ mark, int32_t* cq, unsigned long long* ncq,
                   MsSums sums) {
  const int lane = threadIdx.x & 31;
  unsigned dropped_cols = 0;
  unsigned long long pairs = 0;
  T low = Lim<T>::max();
  for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < npiece;
       i += ((int64_t)gridDim.x * blockDim.x) >> 5) {
    const int4 p = pieces[i];
    const int64_t v = hubs[p.x];
    if (mark && !((__ldcg(mark + (v >> 5)) >> (v & 31)) & 1u)) continue;
    T best = Lim<T>::max();
    const bool any = bs_pull<T>(g, D, chg, chg_next, p.y, p.z, lane, best);
    bool dropped = false;
    if (any) {
      T* dv = D + v * 32 + lane;
      if (best < *dv) dropped = best < b_atomic_min<T>(dv, best);
      if (dropped) {
        low = best < low ? best : low;
        ++pairs;
      }
    }
    const unsigned b = __ballot_sync(kFullB, dropped);
    dropped_cols |= b;
    if (lane == 0 && b) ms_changed(v, b, chg_next, count, cq, ncq);
  }
  if (drop && lane == 0 && dropped_cols) atomicOr(drop, dropped_cols);
  sums.add<T>(pairs, low);
}

}  // namespace
}  // namespace gg
