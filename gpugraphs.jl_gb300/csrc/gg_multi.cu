// gg_multi.cu -- many independent graphs processed by single launches.
//
// A gg_multigraph holds G square CSR graphs concatenated into one block-diagonal
// structure: each graph keeps its own 1-based Int32 column ids, and 64-bit offsets
// locate its rows and entries (the total entry count may exceed Int32).  Vertex v of
// graph g has the global id row_off[g] + v - 1.
//  * gg_multigraph_spmv: y = A_g x_g (plus-times Float32) for every graph in one
//    kernel launch, 8 lanes per row.
//  * gg_multigraph_bfs: one BFS per graph (one source each) in ONE persistent
//    cooperative launch: all graphs advance level by level together, separated by a
//    grid barrier; frontiers are global queues of global vertex ids.  The barrier's
//    wait is bounded: on timeout it records an error, every block returns, and the
//    call reports GG_ERR_TIMEOUT.  The launch (with its resets) is captured once in
//    a CUDA graph and replayed by later calls.
//  * gg_multigraph_sssp: one single-source shortest-path search per graph in one
//    persistent cooperative launch (near-far ordered relaxation, atomic min, bounded
//    grid barrier), captured in a CUDA graph the same way.
//  The captured launches read the result pointer from device memory (the word after the
//  sources), so a call with another result vector replays the same CUDA graph.
// Levels follow bfs_distances (src/algorithms/bfs.jl:1-73): edges with odd / true
// stored values (every stored entry of a floating-point graph, i.e. its Bool
// pattern), dist = hop level, typemax(Int32) when unreached.  Distances follow
// shortest_path (src/algorithms/shortest_path.jl:12-83) for non-negative weights.
// Both searches use the rows of A_T as out-edges, which equals the reference for
// symmetric graphs.
#include <algorithm>
#include <vector>

#include "gg_band.h"
#include "gg_queue.cuh"
#include "gg_semiring.cuh"

struct gg_multigraph {
  int device = 0;
  int64_t ngraphs = 0;
  int64_t total_n = 0, total_nnz = 0;
  int dtype = GG_FLOAT32;
  int64_t* row_off = nullptr;  // [G+1] global vertex offsets (0-based)
  int64_t* rp64 = nullptr;     // [total_n+1] global 0-based entry offsets of each row
  int32_t* colval = nullptr;   // [total_nnz] global 0-based column (vertex) ids
  void* nzval = nullptr;       // [total_nnz]
  std::vector<int64_t> h_row_off;
  bool all_odd = true;
  // persistent BFS state
  unsigned* visited = nullptr;
  int32_t* q[2] = {nullptr, nullptr};
  unsigned long long* ctr = nullptr;  // [3] rotating queue counters, [3] of the far lists
  unsigned* bar = nullptr;  // [8] barrier arrivals, unused, error, levels, poll limit
  int64_t* d_src = nullptr;           // [G + 1] global source ids, address of the results
  unsigned polls_set = 0;  // poll limit last written to bar[4] (0: none yet)
  cudaGraphExec_t gexec = nullptr;
  int grid = 0;
  // persistent shortest-path state (allocated on first use)
  unsigned* inq[2] = {nullptr, nullptr};  // queued vertices of this / the next step
  unsigned* infar = nullptr;              // vertices in the far list
  int32_t* qf[2] = {nullptr, nullptr};    // far lists
  void* sssp_mem = nullptr;               // one allocation behind the five
  double sum_w = 0.0;                     // sum of the stored values (finite ones)
  cudaGraphExec_t sssp_gexec = nullptr;
  int nonneg = -1;  // all stored values >= 0 (and not NaN)? -1: not yet checked
};

// the context's barrier poll limit into bar[4] (kept across launches: the captured
// graphs clear bar[0..3] only)
static int mg_set_polls(gg_ctx* ctx, gg_multigraph* M) {
  const unsigned p = gg::barrier_polls(ctx);
  if (M->polls_set != p) {
    GG_CUDA(cudaMemcpyAsync(M->bar + 4, &p, sizeof(unsigned), cudaMemcpyHostToDevice, ctx->stream));
    GG_CUDA(cudaStreamSynchronize(ctx->stream));
    M->polls_set = p;
  }
  return GG_OK;
}

namespace gg {

static const unsigned kFullM = 0xffffffffu;

// 8 lanes per row over all graphs' rows (global column ids: no per-row graph lookup)
__global__ void __launch_bounds__(256)
    k_mg_spmv(int64_t total_n, const int64_t* __restrict__ rp, const int32_t* __restrict__ colval,
              const float* __restrict__ nz, const float* __restrict__ x, float* __restrict__ y) {
  const int sub = threadIdx.x & 7;
  const unsigned gm = 0xffu << ((threadIdx.x & 31) & ~7);
  for (int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3; r < total_n;
       r += ((int64_t)gridDim.x * blockDim.x) >> 3) {
    float acc = 0.0f;
    const int64_t k1 = rp[r + 1];
    for (int64_t k = rp[r] + sub; k < k1; k += 8)
      acc = __fadd_rn(acc, __fmul_rn(ld_stream(nz + k), __ldg(x + ld_stream(colval + k))));
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) acc = __fadd_rn(acc, __shfl_xor_sync(gm, acc, o, 8));
    if (sub == 0) y[r] = acc;
  }
}

__device__ __forceinline__ bool mg_odd(const void* nz, int tv, int64_t k) {
  switch (tv) {
    case GG_BOOL: return static_cast<const uint8_t*>(nz)[k] & 1;
    case GG_INT32: return static_cast<const int32_t*>(nz)[k] & 1;
    case GG_INT64: return static_cast<const int64_t*>(nz)[k] & 1;
  }
  return false;
}

// Persistent launches: kMgThreads per block; a frontier vertex gets kMgLanes lanes, so a
// warp keeps four vertices' edge loads in flight (a warp per vertex left 13 of 32 lanes
// idle at a mean degree of 19, waited on one vertex's chain at a time, and did one
// atomic on the queue's length for nearly every vertex).  128 random graphs of 1000 to
// 200000 vertices (93 M entries), Int32 shortest paths: 14.4 -> 3.3 ms, together with
// the near-far order; bound by the chain of dependent L2 round trips of its 133 steps
// (48 warps an SM, 24% issue, L2 29%).  4 / 8 / 16 lanes a vertex: 3.7 / 3.25 / 3.4 ms;
// 32 / 48 / 64 warps an SM: 3.7 / 3.25 / 3.3 ms.
static const int kMgThreads = 512;
static const int kMgLanes = 8;
static const int kMgVerts = 32 / kMgLanes;
static const int kMgStep = 2;  // edges in flight per lane

// end of a step: every block's appends are in, the leader waits for all blocks and
// reads the length of the list the next step takes (bar: arrivals, unused, error,
// levels / steps done, poll limit)
struct MgStep {
  long long len, flen;
  int ok;
};
__device__ __forceinline__ bool mg_step_end(MgStep& S, unsigned* bar, unsigned target,
                                            unsigned long long limit, unsigned long long* len,
                                            unsigned long long* flen) {
  __syncthreads();
  if (threadIdx.x == 0) {
    S.ok = coop_leader_sync(bar, target, limit);
    S.len = (long long)*((volatile unsigned long long*)len);
    if (flen) S.flen = (long long)*((volatile unsigned long long*)flen);
  }
  __syncthreads();
  return S.ok;
}

__global__ void k_mg_fill(const int64_t* src, int64_t G, int64_t n, int32_t v) {
  int32_t* d = reinterpret_cast<int32_t*>(src[G]);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    d[i] = v;
}

__global__ void k_mg_bfs_init(int64_t G, const int64_t* src, unsigned* visited, int32_t* q,
                              unsigned long long* ctr) {
  int32_t* dist = reinterpret_cast<int32_t*>(src[G]);
  for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < G;
       g += (int64_t)gridDim.x * blockDim.x) {
    const int64_t v = src[g];
    atomicOr(visited + (v >> 5), 1u << (v & 31));
    dist[v] = 0;
    q[g] = (int32_t)v;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    ctr[0] = (unsigned long long)G;  // queue size of level 0
    ctr[1] = 0;
    ctr[2] = 0;
  }
}

// all graphs' BFS levels in one persistent launch
__global__ void __launch_bounds__(kMgThreads, 3)
    k_mg_bfs(int64_t G, const int64_t* __restrict__ src, const int64_t* __restrict__ rp,
             const int32_t* __restrict__ colval, const void* nz, int tv, int odd_only,
             unsigned* visited, int32_t* qa, int32_t* qb, unsigned long long* ctr, unsigned* bar) {
  __shared__ int32_t stage[kMgThreads / 32][WarpQueue::kCap];
  __shared__ MgStep S;
  int32_t* dist = reinterpret_cast<int32_t*>(src[G]);
  const unsigned long long limit = bar[4];  // written by the host before each launch
  const int lane = threadIdx.x & 31;
  const int64_t gw = (int64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x;
  const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
  int32_t* cur = qa;
  int32_t* nxt = qb;
  long long nf = (long long)*((volatile unsigned long long*)ctr);
  for (int32_t level = 1;; ++level) {
    const int r = level % 3;
    if (nf == 0) {
      if (blockIdx.x == 0 && threadIdx.x == 0) bar[3] = (unsigned)(level - 1);
      return;
    }
    // counter for this level's appends was zeroed two levels ago; zero the next one
    if (blockIdx.x == 0 && threadIdx.x == 0) ctr[(r + 1) % 3] = 0;
    WarpQueue wq(stage[threadIdx.x >> 5], nxt, ctr + r);
    for (int64_t i0 = gw * kMgVerts; i0 < nf; i0 += nw * kMgVerts) {
      const int64_t i = i0 + lane / kMgLanes;
      int64_t k = 0, k1 = 0;
      if (i < nf) {
        const int64_t v = __ldcg(cur + i);
        k = rp[v] + lane % kMgLanes;
        k1 = rp[v + 1];
      }
      while (__any_sync(kFullM, k < k1)) {
        int32_t w[kMgStep];
        unsigned seen[kMgStep];
#pragma unroll
        for (int t = 0; t < kMgStep; ++t) {
          const int64_t kk = k + t * kMgLanes;
          w[t] = kk < k1 && (!odd_only || mg_odd(nz, tv, kk)) ? __ldg(colval + kk) : -1;
        }
#pragma unroll
        for (int t = 0; t < kMgStep; ++t) seen[t] = w[t] >= 0 ? __ldcg(visited + (w[t] >> 5)) : ~0u;
#pragma unroll
        for (int t = 0; t < kMgStep; ++t) {
          const unsigned bit = 1u << (w[t] & 31);
          const bool claim = !(seen[t] & bit) && !(atomicOr(visited + (w[t] >> 5), bit) & bit);
          if (claim) dist[w[t]] = level;
          wq.push(claim, w[t]);
        }
        k += kMgStep * kMgLanes;
      }
    }
    wq.flush();
    if (!mg_step_end(S, bar, (unsigned)level * gridDim.x, limit, ctr + r, nullptr)) return;
    nf = S.len;
    int32_t* t = cur;
    cur = nxt;
    nxt = t;
  }
}

template <typename T> __device__ __forceinline__ T mg_atomic_min(T* p, T v);
template <> __device__ __forceinline__ int32_t mg_atomic_min<int32_t>(int32_t* p, int32_t v) {
  return atomicMin(p, v);
}
template <> __device__ __forceinline__ int64_t mg_atomic_min<int64_t>(int64_t* p, int64_t v) {
  return (int64_t)atomicMin((long long*)p, (long long)v);
}
// distances are non-negative and never -0.0 (+0.0 + w), so floats order like their bits
template <> __device__ __forceinline__ float mg_atomic_min<float>(float* p, float v) {
  return __int_as_float(atomicMin((int*)p, __float_as_int(v)));
}
template <> __device__ __forceinline__ double mg_atomic_min<double>(double* p, double v) {
  return __longlong_as_double(atomicMin((long long*)p, __double_as_longlong(v)));
}

template <typename T>
__device__ __forceinline__ T mg_weight(const void* nz, int tv, int64_t k) {
  switch (tv) {
    case GG_BOOL: return static_cast<T>(static_cast<const uint8_t*>(nz)[k]);
    case GG_INT32: return static_cast<T>(static_cast<const int32_t*>(nz)[k]);
    case GG_INT64: return static_cast<T>(static_cast<const int64_t*>(nz)[k]);
    case GG_FLOAT32: return static_cast<T>(static_cast<const float*>(nz)[k]);
  }
  return static_cast<T>(static_cast<const double*>(nz)[k]);
}

template <typename T>
__global__ void k_mg_fill_t(const int64_t* src, int64_t G, int64_t n, T v) {
  T* d = reinterpret_cast<T*>(src[G]);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    d[i] = v;
}

template <typename T>
__global__ void k_mg_sssp_seed(int64_t G, const int64_t* src, unsigned* inq, int32_t* q,
                               unsigned long long* ctr) {
  T* dist = reinterpret_cast<T*>(src[G]);
  for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < G;
       g += (int64_t)gridDim.x * blockDim.x) {
    const int64_t v = src[g];
    dist[v] = T(0);
    atomicOr(inq + (v >> 5), 1u << (v & 31));
    q[g] = (int32_t)v;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    ctr[0] = (unsigned long long)G;
    for (int i = 1; i < 6; ++i) ctr[i] = 0;
  }
}

// All graphs' shortest paths in one persistent launch, near-far ordered over all graphs
// together: vertices below the distance threshold thr are relaxed, improved vertices at
// or above it wait in a far list, and when no near vertex is left thr grows by delta and
// the far list is split.  The fixpoint is the same (every improved vertex is relaxed
// again, and distances only fall), but a vertex is relaxed little more than once instead
// of once per improvement.  icur / inxt mark queued vertices, infar the waiting ones.
// Band b appends to far list b mod 2 counted in fctr[b mod 3]; every step zeroes the
// counter that the band after next will use.
template <typename T>
__global__ void __launch_bounds__(kMgThreads, 3)
    k_mg_sssp(int64_t G, const int64_t* __restrict__ src, const int64_t* __restrict__ rp,
              const int32_t* __restrict__ colval, const void* nz, int tv, unsigned* inq_a,
              unsigned* inq_b, unsigned* infar, int32_t* qa, int32_t* qb, int32_t* fa, int32_t* fb,
              unsigned long long* ctr, unsigned* bar, T delta, int64_t max_steps) {
  __shared__ int32_t stage[2][kMgThreads / 32][WarpQueue::kCap];
  __shared__ MgStep S;
  T* dist = reinterpret_cast<T*>(src[G]);
  unsigned long long* fctr = ctr + 3;
  const unsigned long long limit = bar[4];  // written by the host before each launch
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t gw = (int64_t)warp * gridDim.x + blockIdx.x;
  const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
  int32_t* cur = qa;
  int32_t* nxt = qb;
  unsigned* icur = inq_a;
  unsigned* inxt = inq_b;
  T thr = delta, width = delta;
  int64_t band = 0;
  bool was_change = false;
  int64_t empty = 0;  // bands that moved nothing, so far
  int run = 0;        // the latest ones in a row
  long long nf = (long long)*((volatile unsigned long long*)ctr), nfar = 0;
  for (int64_t step = 1;; ++step) {
    const int r = (int)(step % 3);
    // counted here, not where a band moves: there the kernel spills at its 40 registers (128
    // graphs at once 3.26 -> 3.33 ms)
    run = nf == 0 && was_change ? run + 1 : 0;
    empty += run > 0;
    const bool out = step - empty > max_steps || run > kEmptyBandRun;
    if ((nf == 0 && nfar == 0) || out) {
      if (blockIdx.x == 0 && threadIdx.x == 0) {
        bar[3] = (unsigned)(step - 1);
        if (out) atomicExch(bar + 2, 2u);  // still improving
      }
      return;
    }
    int fc = (int)(band % 3);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      ctr[(r + 1) % 3] = 0;
      fctr[(fc + 2) % 3] = 0;
    }
    WarpQueue wn(stage[0][warp], nxt, ctr + r);
    if (nf == 0) {
      const int32_t* from = band % 2 ? fb : fa;
      ++band;
      fc = (int)(band % 3);
      WarpQueue wf(stage[1][warp], band % 2 ? fb : fa, fctr + fc);
      // an empty band doubles the next one: gaps between the distances (or a width below
      // a large threshold's rounding) cost a logarithmic number of steps
      width = !was_change ? delta : (width < Lim<T>::max() / 2 ? w_add(width, width) : width);
      was_change = true;
      thr = thr > Lim<T>::max() - width ? Lim<T>::max() : w_add(thr, width);
      for (int64_t i0 = gw * 32; i0 < nfar; i0 += nw * 32) {
        const int64_t i = i0 + lane;
        bool to_near = false, to_far = false;
        int32_t v = 0;
        if (i < nfar) {
          v = __ldcg(from + i);
          if (__ldcg(dist + v) < thr) {
            const unsigned bit = 1u << (v & 31);
            atomicAnd(infar + (v >> 5), ~bit);
            to_near = !(atomicOr(inxt + (v >> 5), bit) & bit);
          } else {
            to_far = true;
          }
        }
        wn.push(to_near, v);
        wf.push(to_far, v);
      }
      wf.flush();
    } else {
      was_change = false;
      WarpQueue wf(stage[1][warp], band % 2 ? fb : fa, fctr + fc);
      for (int64_t i0 = gw * kMgVerts; i0 < nf; i0 += nw * kMgVerts) {
        const int64_t i = i0 + lane / kMgLanes;
        int64_t k = 0, k1 = 0;
        T du = T(0);
        if (i < nf) {
          const int64_t u = __ldcg(cur + i);
          if (lane % kMgLanes == 0) atomicAnd(icur + (u >> 5), ~(1u << (u & 31)));
          k = rp[u] + lane % kMgLanes;
          k1 = rp[u + 1];
          du = __ldcg(dist + u);
        }
        while (__any_sync(kFullM, k < k1)) {
          int32_t v[kMgStep];
          T cand[kMgStep], dv[kMgStep];
#pragma unroll
          for (int t = 0; t < kMgStep; ++t) {
            const int64_t kk = k + t * kMgLanes;
            v[t] = kk < k1 ? __ldg(colval + kk) : -1;
            const T w = kk < k1 ? mg_weight<T>(nz, tv, kk) : Lim<T>::max();
            cand[t] = (w == Lim<T>::max() || du == Lim<T>::max()) ? Lim<T>::max() : w_add(w, du);
          }
#pragma unroll
          for (int t = 0; t < kMgStep; ++t) dv[t] = v[t] >= 0 ? __ldcg(dist + v[t]) : Lim<T>::min();
          unsigned near_add = 0, far_add = 0;  // bit t
#pragma unroll
          for (int t = 0; t < kMgStep; ++t)
            if (cand[t] < dv[t] && cand[t] < mg_atomic_min<T>(dist + v[t], cand[t])) {
              const unsigned bit = 1u << (v[t] & 31);
              if (cand[t] < thr) near_add |= !(atomicOr(inxt + (v[t] >> 5), bit) & bit) ? 1u << t : 0u;
              else far_add |= !(atomicOr(infar + (v[t] >> 5), bit) & bit) ? 1u << t : 0u;
            }
          if (__any_sync(kFullM, near_add | far_add)) {
#pragma unroll
            for (int t = 0; t < kMgStep; ++t) {
              wn.push((near_add >> t) & 1u, v[t]);
              wf.push((far_add >> t) & 1u, v[t]);
            }
          }
          k += kMgStep * kMgLanes;
        }
      }
      wf.flush();
    }
    wn.flush();
    if (!mg_step_end(S, bar, (unsigned)step * gridDim.x, limit, ctr + r, fctr + fc)) return;
    nf = S.len;
    nfar = S.flen;
    int32_t* t = cur;
    cur = nxt;
    nxt = t;
    unsigned* tb = icur;
    icur = inxt;
    inxt = tb;
  }
}

// stored values: any negative or NaN one (*bad), and the sum of the finite ones
__global__ void k_mg_values(const void* nz, int tv, int64_t nnz, unsigned* bad, double* sum) {
  unsigned b = 0;
  double s = 0.0;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < nnz;
       k += (int64_t)gridDim.x * blockDim.x) {
    const double w = mg_weight<double>(nz, tv, k);
    b |= !(w >= 0.0);
    if (w <= 1.7976931348623157e308) s += w;
  }
  if (__syncthreads_or(b) && threadIdx.x == 0) atomicOr(bad, 1u);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(kFullM, s, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(sum, s);
}

// global 0-based column ids: colval_g (1-based within graph g) + row_off[g] - 1
__global__ void k_mg_cols(int64_t nnz, const int32_t* __restrict__ cv, int32_t base, int32_t* out) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < nnz;
       k += (int64_t)gridDim.x * blockDim.x)
    out[k] = cv[k] - 1 + base;
}

// global entry offsets of each row: rp64[row_off[g] + v] = nnz_off[g] + rowptr_g[v] - 1
__global__ void k_mg_rp(int64_t n, const int32_t* rp_local, int64_t row_base, int64_t nnz_base,
                        int64_t* rp64) {
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v <= n;
       v += (int64_t)gridDim.x * blockDim.x)
    rp64[row_base + v] = nnz_base + (int64_t)rp_local[v] - 1;
}

static int mg_grid(int num_sms, int64_t work) {
  int64_t g = (work + 255) / 256;
  const int64_t cap = (int64_t)num_sms * 8;
  return (int)(g > cap ? cap : (g < 1 ? 1 : g));
}

}  // namespace gg

using namespace gg;

// checks the sources and puts their global ids, then the address of the results, into
// the words the captured launches read
static int mg_upload_sources(gg_ctx* ctx, gg_multigraph* M, const int64_t* sources, void* dist) {
  std::vector<int64_t> gsrc(M->ngraphs + 1);
  for (int64_t g = 0; g < M->ngraphs; ++g) {
    const int64_t n = M->h_row_off[g + 1] - M->h_row_off[g];
    if (sources[g] < 1 || sources[g] > n)
      return set_error(GG_ERR_BOUNDS, "source %lld of graph %lld out of 1:%lld", (long long)sources[g],
                       (long long)g, (long long)n);
    gsrc[g] = M->h_row_off[g] + sources[g] - 1;
  }
  gsrc[M->ngraphs] = (int64_t)(uintptr_t)dist;
  GG_CUDA(cudaMemcpyAsync(M->d_src, gsrc.data(), gsrc.size() * sizeof(int64_t),
                          cudaMemcpyHostToDevice, ctx->stream));
  return GG_OK;
}

extern "C" {

int gg_multigraph_create(gg_ctx* ctx, const gg_mat* const* graphs, int64_t ngraphs,
                         gg_multigraph** out) {
  if (!ctx || !graphs || !out || ngraphs < 1) return set_error(GG_ERR_ARGUMENT, "bad arguments");
  *out = nullptr;
  GG_CUDA(cudaSetDevice(ctx->device));
  const int dt = graphs[0]->dtype;
  std::vector<int64_t> off(ngraphs + 1, 0), noff(ngraphs + 1, 0);
  for (int64_t g = 0; g < ngraphs; ++g) {
    const gg_mat* A = graphs[g];
    if (!A || A->format != GG_FMT_CSR) return set_error(GG_ERR_ARGUMENT, "graph %lld is not a CSR handle", (long long)g);
    if (A->m != A->n) return set_error(GG_ERR_DIMENSION, "graph %lld is not square", (long long)g);
    if (A->dtype != dt) return set_error(GG_ERR_TYPE, "all graphs must share one element type");
    off[g + 1] = off[g] + A->m;
    noff[g + 1] = noff[g] + A->nnz;
  }
  if (off[ngraphs] >= INT32_MAX) return set_error(GG_ERR_ARGUMENT, "more than 2^31 vertices in total");
  gg_multigraph* M = new gg_multigraph();
  M->device = ctx->device;
  M->ngraphs = ngraphs;
  M->total_n = off[ngraphs];
  M->total_nnz = noff[ngraphs];
  M->dtype = dt;
  M->h_row_off = off;
  const size_t esz = dtype_size(dt);
  cudaError_t e = cudaMalloc((void**)&M->row_off, (ngraphs + 1) * sizeof(int64_t));
  if (e == cudaSuccess) e = cudaMalloc((void**)&M->rp64, (M->total_n + 1) * sizeof(int64_t));
  if (e == cudaSuccess) e = cudaMalloc((void**)&M->colval, (M->total_nnz + 1) * sizeof(int32_t));
  if (e == cudaSuccess) e = cudaMalloc(&M->nzval, (M->total_nnz + 1) * esz);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(M->row_off, off.data(), (ngraphs + 1) * sizeof(int64_t),
                        cudaMemcpyHostToDevice, ctx->stream);
  for (int64_t g = 0; g < ngraphs && e == cudaSuccess; ++g) {
    const gg_mat* A = graphs[g];
    k_mg_rp<<<mg_grid(ctx->num_sms, A->m + 1), 256, 0, ctx->stream>>>(A->m, A->rowptr, off[g], noff[g],
                                                                       M->rp64);
    e = cudaGetLastError();
    if (e == cudaSuccess && A->nnz > 0) {
      k_mg_cols<<<mg_grid(ctx->num_sms, A->nnz), 256, 0, ctx->stream>>>(A->nnz, A->colval,
                                                                        (int32_t)off[g], M->colval + noff[g]);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess && A->nnz > 0)
      e = cudaMemcpyAsync(static_cast<char*>(M->nzval) + noff[g] * esz, A->nzval, A->nnz * esz,
                          cudaMemcpyDeviceToDevice, ctx->stream);
  }
  // BFS state
  const int64_t nw = M->total_n / 32 + 2;
  if (e == cudaSuccess) e = cudaMalloc((void**)&M->visited, nw * sizeof(unsigned));
  if (e == cudaSuccess) e = cudaMalloc((void**)&M->q[0], (M->total_n + 1) * sizeof(int32_t));
  if (e == cudaSuccess) e = cudaMalloc((void**)&M->q[1], (M->total_n + 1) * sizeof(int32_t));
  if (e == cudaSuccess) e = cudaMalloc((void**)&M->ctr, 8 * sizeof(unsigned long long));
  if (e == cudaSuccess) e = cudaMalloc((void**)&M->bar, 8 * sizeof(unsigned));
  if (e == cudaSuccess) e = cudaMemset(M->bar, 0, 8 * sizeof(unsigned));
  if (e == cudaSuccess) e = cudaMalloc((void**)&M->d_src, (ngraphs + 1) * sizeof(int64_t));
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  if (e != cudaSuccess) {
    gg_multigraph_destroy(M);
    return cuda_error(e, "gg_multigraph_create");
  }
  // edge activity for the levels semiring: odd / true values only
  if (dt == GG_BOOL || dt == GG_INT32 || dt == GG_INT64) {
    M->all_odd = true;  // checked lazily by the kernel's odd_only flag below
  }
  *out = M;
  return GG_OK;
}

int gg_multigraph_destroy(gg_multigraph* M) {
  if (!M) return GG_OK;
  cudaSetDevice(M->device);
  if (M->gexec) cudaGraphExecDestroy(M->gexec);
  if (M->sssp_gexec) cudaGraphExecDestroy(M->sssp_gexec);
  cudaFree(M->sssp_mem);
  cudaFree(M->row_off);
  cudaFree(M->rp64);
  cudaFree(M->colval);
  cudaFree(M->nzval);
  cudaFree(M->visited);
  cudaFree(M->q[0]);
  cudaFree(M->q[1]);
  cudaFree(M->ctr);
  cudaFree(M->bar);
  cudaFree(M->d_src);
  delete M;
  return GG_OK;
}

int gg_multigraph_info(const gg_multigraph* M, int64_t* ngraphs, int64_t* total_n,
                       int64_t* total_nnz, int64_t* row_offsets) {
  if (!M) return set_error(GG_ERR_ARGUMENT, "NULL multigraph");
  if (ngraphs) *ngraphs = M->ngraphs;
  if (total_n) *total_n = M->total_n;
  if (total_nnz) *total_nnz = M->total_nnz;
  if (row_offsets)
    for (int64_t g = 0; g <= M->ngraphs; ++g) row_offsets[g] = M->h_row_off[g];
  return GG_OK;
}

int gg_multigraph_spmv(gg_ctx* ctx, const gg_multigraph* M, const float* x, float* y) {
  if (!ctx || !M || !x || !y) return set_error(GG_ERR_ARGUMENT, "NULL argument");
  if (M->dtype != GG_FLOAT32) return set_error(GG_ERR_TYPE, "multigraph SpMV needs Float32 values");
  GG_CUDA(cudaSetDevice(ctx->device));
  k_mg_spmv<<<mg_grid(ctx->num_sms, M->total_n * 8), 256, 0, ctx->stream>>>(
      M->total_n, M->rp64, M->colval, static_cast<const float*>(M->nzval), x, y);
  GG_CUDA(cudaGetLastError());
  return GG_OK;
}

int gg_multigraph_bfs(gg_ctx* ctx, gg_multigraph* M, const int64_t* sources, int32_t* dist,
                      int64_t* levels_out) {
  if (!ctx || !M || !sources || !dist) return set_error(GG_ERR_ARGUMENT, "NULL argument");
  GG_CUDA(cudaSetDevice(ctx->device));
  GG_CHECK(mg_upload_sources(ctx, M, sources, dist));
  if (!M->gexec) {
    int per_sm = 0;
    GG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_mg_bfs, kMgThreads, 0));
    if (per_sm < 1) return set_error(GG_ERR_CUDA, "k_mg_bfs cannot be resident");
    M->grid = ctx->num_sms * per_sm;  // every block resident: the cooperative barrier is safe
    cudaStream_t cs = nullptr;
    GG_CUDA(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
    cudaGraph_t graph = nullptr;
    cudaError_t e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
    const int64_t nw = M->total_n / 32 + 2;
    const int odd_only = dtype_is_float(M->dtype) ? 0 : 1;  // floats: the Bool pattern
    int64_t G = M->ngraphs;
    if (e == cudaSuccess) e = cudaMemsetAsync(M->visited, 0, nw * sizeof(unsigned), cs);
    if (e == cudaSuccess) e = cudaMemsetAsync(M->bar, 0, 4 * sizeof(unsigned), cs);
    if (e == cudaSuccess) {
      k_mg_fill<<<mg_grid(ctx->num_sms, M->total_n), 256, 0, cs>>>(M->d_src, G, M->total_n, INT32_MAX);
      k_mg_bfs_init<<<mg_grid(ctx->num_sms, G), 256, 0, cs>>>(G, M->d_src, M->visited, M->q[0], M->ctr);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess) {
      int tv = M->dtype;
      void* args[] = {&G, &M->d_src, &M->rp64, &M->colval, &M->nzval, &tv, (void*)&odd_only,
                      &M->visited, &M->q[0], &M->q[1], &M->ctr, &M->bar};
      e = cudaLaunchCooperativeKernel((const void*)k_mg_bfs, dim3(M->grid), dim3(kMgThreads), args, 0,
                                      cs);
    }
    cudaError_t e2 = cudaStreamEndCapture(cs, &graph);
    if (e == cudaSuccess) e = e2;
    if (e == cudaSuccess) e = cudaGraphInstantiate(&M->gexec, graph, 0);
    if (graph) cudaGraphDestroy(graph);
    cudaStreamDestroy(cs);
    if (e != cudaSuccess) return cuda_error(e, "multigraph BFS graph capture");
  }
  GG_CHECK(mg_set_polls(ctx, M));
  GG_CUDA(cudaGraphLaunch(M->gexec, ctx->stream));
  unsigned hb[4] = {0, 0, 0, 0};
  GG_CUDA(cudaMemcpyAsync(hb, M->bar, sizeof(hb), cudaMemcpyDeviceToHost, ctx->stream));
  GG_CUDA(cudaStreamSynchronize(ctx->stream));
  if (hb[2]) return set_error(GG_ERR_TIMEOUT, "multigraph BFS barrier wait ran out");
  if (levels_out) *levels_out = hb[3];
  return GG_OK;
}

}  // extern "C"

// Near-far band: this multiple of the mean weight over the mean degree (the distances of
// random graphs go as that), and at least 1 for whole-number weights.  Narrow bands cost
// steps, wide ones repeat relaxations: 2 / 8 / 16 / 32 / 64 gave 476 / 201 / 133 / 91 / -
// steps and 5.0 / 3.5 / 3.25 / 4.1 / 4.6 ms on the 128 graphs above.  Fewer entries than
// kMgBandNnz run as plain rounds (one band): repeated relaxations of a small frontier
// fit the same latency-bound step.  Bands / plain rounds, ms: 0.30 M entries 0.43 / 0.22,
// 3 M 0.71 / 0.42, 8 M 1.22 / 0.99, 15 M 1.15 / 0.86, 93 M 3.25 / 4.40.
static const double kMgBand = 16.0;
static const int64_t kMgBandNnz = 1 << 25;

template <typename T>
static int mg_sssp_capture(gg_ctx* ctx, gg_multigraph* M) {
  int per_sm = 0;
  GG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_mg_sssp<T>, kMgThreads, 0));
  if (per_sm < 1) return set_error(GG_ERR_CUDA, "k_mg_sssp cannot be resident");
  const int grid = ctx->num_sms * per_sm;  // every block resident: the barrier is safe
  const double nnz = M->total_nnz > 0 ? (double)M->total_nnz : 1.0;
  T delta = band_width<T>(kMgBand * (M->sum_w / nnz) /
                           (nnz / (double)(M->total_n > 0 ? M->total_n : 1)));
  if (M->total_nnz < kMgBandNnz) delta = Lim<T>::max();
  cudaStream_t cs = nullptr;
  GG_CUDA(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
  cudaGraph_t graph = nullptr;
  cudaError_t e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
  const int64_t nw = M->total_n / 32 + 2;
  int64_t G = M->ngraphs;
  int64_t max_steps = 8 * M->total_n + 1024;
  if (e == cudaSuccess) e = cudaMemsetAsync(M->inq[0], 0, nw * sizeof(unsigned), cs);
  if (e == cudaSuccess) e = cudaMemsetAsync(M->inq[1], 0, nw * sizeof(unsigned), cs);
  if (e == cudaSuccess) e = cudaMemsetAsync(M->infar, 0, nw * sizeof(unsigned), cs);
  if (e == cudaSuccess) e = cudaMemsetAsync(M->bar, 0, 4 * sizeof(unsigned), cs);
  if (e == cudaSuccess) {
    k_mg_fill_t<T><<<mg_grid(ctx->num_sms, M->total_n), 256, 0, cs>>>(M->d_src, G, M->total_n,
                                                                      Lim<T>::max());
    k_mg_sssp_seed<T><<<mg_grid(ctx->num_sms, G), 256, 0, cs>>>(G, M->d_src, M->inq[0], M->q[0], M->ctr);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) {
    int tv = M->dtype;
    void* args[] = {&G, &M->d_src, &M->rp64, &M->colval, &M->nzval, &tv, &M->inq[0], &M->inq[1],
                    &M->infar, &M->q[0], &M->q[1], &M->qf[0], &M->qf[1], &M->ctr, &M->bar, &delta,
                    &max_steps};
    e = cudaLaunchCooperativeKernel((const void*)k_mg_sssp<T>, dim3(grid), dim3(kMgThreads), args, 0,
                                    cs);
  }
  cudaError_t e2 = cudaStreamEndCapture(cs, &graph);
  if (e == cudaSuccess) e = e2;
  if (e == cudaSuccess) e = cudaGraphInstantiate(&M->sssp_gexec, graph, 0);
  if (graph) cudaGraphDestroy(graph);
  cudaStreamDestroy(cs);
  if (e != cudaSuccess) return cuda_error(e, "multigraph shortest-path graph capture");
  return GG_OK;
}

extern "C" {

int gg_multigraph_sssp(gg_ctx* ctx, gg_multigraph* M, const int64_t* sources, void* dist,
                       int dist_dtype, int64_t* rounds_out) {
  if (!ctx || !M || !sources || !dist) return set_error(GG_ERR_ARGUMENT, "NULL argument");
  const int want = M->dtype == GG_BOOL ? GG_INT32 : M->dtype;
  if (dist_dtype != want)
    return set_error(GG_ERR_TYPE, "dist element type must be Int32 for Bool graphs, else the graphs' type");
  GG_CUDA(cudaSetDevice(ctx->device));
  if (M->nonneg < 0) {
    double* dsum = reinterpret_cast<double*>(ctx->d_flags + 2);
    GG_CUDA(cudaMemsetAsync(ctx->d_flags, 0, 4 * sizeof(unsigned), ctx->stream));
    k_mg_values<<<mg_grid(ctx->num_sms, M->total_nnz), 256, 0, ctx->stream>>>(
        M->nzval, M->dtype, M->total_nnz, ctx->d_flags, dsum);
    GG_CUDA(cudaGetLastError());
    GG_CUDA(cudaMemcpyAsync(ctx->h_flags, ctx->d_flags, 4 * sizeof(unsigned), cudaMemcpyDeviceToHost,
                            ctx->stream));
    GG_CUDA(cudaStreamSynchronize(ctx->stream));
    M->nonneg = ctx->h_flags[0] ? 0 : 1;
    M->sum_w = *reinterpret_cast<const double*>(ctx->h_flags + 2);
  }
  if (!M->nonneg)
    return set_error(GG_ERR_UNSUPPORTED, "multigraph shortest paths need non-negative weights");
  const int64_t nw = M->total_n / 32 + 2;
  if (!M->sssp_mem) {
    const size_t bm = ((size_t)nw * sizeof(unsigned) + 255) & ~(size_t)255;
    const size_t qb = ((size_t)(M->total_n + 1) * sizeof(int32_t) + 255) & ~(size_t)255;
    GG_CUDA(cudaMalloc(&M->sssp_mem, 3 * bm + 2 * qb));
    char* p = static_cast<char*>(M->sssp_mem);
    M->inq[0] = (unsigned*)p;
    M->inq[1] = (unsigned*)(p + bm);
    M->infar = (unsigned*)(p + 2 * bm);
    M->qf[0] = (int32_t*)(p + 3 * bm);
    M->qf[1] = (int32_t*)(p + 3 * bm + qb);
  }
  GG_CHECK(mg_upload_sources(ctx, M, sources, dist));
  if (!M->sssp_gexec) {
    switch (dist_dtype) {
      case GG_INT32: GG_CHECK(mg_sssp_capture<int32_t>(ctx, M)); break;
      case GG_INT64: GG_CHECK(mg_sssp_capture<int64_t>(ctx, M)); break;
      case GG_FLOAT32: GG_CHECK(mg_sssp_capture<float>(ctx, M)); break;
      default: GG_CHECK(mg_sssp_capture<double>(ctx, M)); break;
    }
  }
  GG_CHECK(mg_set_polls(ctx, M));
  GG_CUDA(cudaGraphLaunch(M->sssp_gexec, ctx->stream));
  unsigned hb[4] = {0, 0, 0, 0};
  GG_CUDA(cudaMemcpyAsync(hb, M->bar, sizeof(hb), cudaMemcpyDeviceToHost, ctx->stream));
  GG_CUDA(cudaStreamSynchronize(ctx->stream));
  if (hb[2] == 1) return set_error(GG_ERR_TIMEOUT, "multigraph shortest-path barrier wait ran out");
  if (hb[2] == 2) return set_error(GG_ERR_NOT_CONVERGED, "multigraph shortest paths did not converge");
  if (rounds_out) *rounds_out = hb[3];
  return GG_OK;
}

}  // extern "C"
