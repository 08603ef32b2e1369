// gg_spmv_kernels.cuh -- SpMV kernels of any semiring policy, and their launches:
// row blocks of a CSR matrix (k_csr_rowblock) and slices of a SELL matrix (k_sell).
// gg_spmv.cu instantiates them for runtime operators and types (SRGen),
// gg_spmv_typed.cu for the common semirings with both fixed (SRTyped).
#pragma once

#include "gg_semiring.cuh"

namespace gg {

static const unsigned kFull = 0xffffffffu;

__device__ __forceinline__ unsigned group_mask(int G) {
  if (G >= 32) return kFull;
  int lane = threadIdx.x & 31;
  return ((1u << G) - 1u) << (lane & ~(G - 1));
}

template <typename T>
__device__ __forceinline__ T shfl_xor_m(unsigned mask, T v, int off, int width) {
  return __shfl_xor_sync(mask, v, off, width);
}
template <typename T>
__device__ __forceinline__ T shfl_idx_m(unsigned mask, T v, int src) {
  return __shfl_sync(mask, v, src);
}
template <>
__device__ __forceinline__ uint8_t shfl_idx_m<uint8_t>(unsigned mask, uint8_t v, int src) {
  return static_cast<uint8_t>(__shfl_sync(mask, static_cast<int>(v), src));
}
template <>
__device__ __forceinline__ uint8_t shfl_xor_m<uint8_t>(unsigned mask, uint8_t v, int off,
                                                       int width) {
  return static_cast<uint8_t>(__shfl_xor_sync(mask, static_cast<int>(v), off, width));
}

// ---------------------------------------------------------------------------------
// storage-order refold with the reference's early exit (csr_spmv_kernel!,
// src/spmv/CSR.jl:47-52) for rows reduced in parallel
//
// A parallel (tree-ordered) fold of a floating-point row differs from the sequential
// fold with its stop at the absorbing value only through NaN: a NaN or -Inf term
// after the sum reached +Inf (GPUGraphs_add), or a NaN after -Inf / +Inf (min /
// max).  Without the stop those give NaN; any other non-finite or finite result is
// the same.  So a row whose parallel result is NaN is folded again, by the whole
// warp: lanes compute 32 products at once (coalesced loads) and the sum is taken in
// storage order through shuffles, stopping where the reference stops.  Integer and
// Bool accumulators never compare unequal to themselves, so they skip this.
// ---------------------------------------------------------------------------------
template <class SR>
__device__ __forceinline__ typename SR::T warp_refold_row(const SR& sr, const int32_t* __restrict__ rowptr,
                                                          const int32_t* __restrict__ colval,
                                                          int64_t row0, int lane) {
  typedef typename SR::T T;
  const int32_t kb = __ldg(rowptr + row0) - 1, ke = __ldg(rowptr + row0 + 1) - 1;
  T acc = sr.neutral();
  bool done = false;
  for (int32_t base = kb; base < ke && !done; base += 32) {
    const int32_t k = base + lane;
    T p = sr.neutral();
    if (k < ke) p = sr.mulk(k, __ldg(colval + k), row0 + 1);
    const int cnt = ke - base < 32 ? ke - base : 32;
    for (int j = 0; j < cnt; ++j) {
      acc = sr.addv(acc, shfl_idx_m<T>(kFull, p, j));
      if (sr.is_absorb(acc)) {
        done = true;
        break;
      }
    }
  }
  return acc;
}

// ---------------------------------------------------------------------------------
// row-block kernel (unmasked CSR)
// ---------------------------------------------------------------------------------
static const int kRBWarps = 8;  // warps per CTA

// Row filter of the masked / range variants (CSR.jl:117-144, :224-313): a row is
// computed when it lies in [lo, hi) (0-based) and mask[row] != 0.
struct RowFilter {
  const void* mask;
  int tmask;
  int64_t lo, hi;
  __device__ __forceinline__ bool keep(int64_t r) const {
    if (r < lo || r >= hi) return false;
    return !mask || !raw_is_zero(load_raw(mask, tmask, r), tmask);
  }
};

// row of stored entry k inside rows [r0, r1) (binary search; only index operators
// that read the row id need it during staging)
__device__ __forceinline__ int64_t row_of(const int32_t* rowptr, int32_t r0, int32_t r1, int32_t k) {
  int32_t lo = r0, hi = r1 - 1;
  while (lo < hi) {
    const int32_t mid = (lo + hi + 1) >> 1;
    if (__ldg(rowptr + mid) - 1 <= k) lo = mid; else hi = mid - 1;
  }
  return lo;
}

template <class SR, bool kFiltered, bool kNeedsRow>
__global__ void __launch_bounds__(kRBWarps * 32)
    k_csr_rowblock(SR sr, const int32_t* __restrict__ rowptr, const int32_t* __restrict__ colval,
                   const int4* __restrict__ blocks, int64_t nblocks, const int4* __restrict__ segs,
                   int64_t nsegs, const int32_t* __restrict__ long_first_seg,
                   const int32_t* __restrict__ long_rows, unsigned int* long_count,
                   typename SR::T* partials, RowFilter flt) {
  typedef typename SR::T T;
  __shared__ T stage[kRBWarps][kBlockNnz];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t nw = (int64_t)gridDim.x * kRBWarps;
  T* st = stage[warp];
  for (int64_t item = (int64_t)blockIdx.x * kRBWarps + warp; item < nblocks + nsegs; item += nw) {
    if (item < nblocks) {
      const int4 b = blocks[item];
      if (kFiltered && (b.y <= flt.lo || b.x >= flt.hi)) continue;
      const int32_t k0 = b.z, k1 = b.w;
      // stage products: 8 independent coalesced loads in flight per lane
      T v[kBlockNnz / 32];
#pragma unroll
      for (int u = 0; u < kBlockNnz / 32; ++u) {
        const int32_t k = k0 + u * 32 + lane;
        if (k < k1)
          v[u] = sr.mulk(k, __ldcs(colval + k), kNeedsRow ? row_of(rowptr, b.x, b.y, k) + 1 : 0);
      }
#pragma unroll
      for (int u = 0; u < kBlockNnz / 32; ++u) {
        const int32_t k = k0 + u * 32 + lane;
        if (k < k1) st[u * 32 + lane] = v[u];
      }
      __syncwarp();
      for (int32_t r = b.x + lane; r < b.y; r += 32) {
        if (kFiltered && !flt.keep(r)) continue;
        const int32_t s = __ldg(rowptr + r) - 1 - k0;
        const int32_t e = __ldg(rowptr + r + 1) - 1 - k0;
        T acc = sr.neutral();
        for (int32_t i = s; i < e; ++i) {
          acc = sr.addv(acc, st[i]);
          if (SR::kHasAbsorbCheck && sr.is_absorb(acc)) break;
        }
        sr.write(r, acc);
      }
      __syncwarp();
    } else {
      const int64_t si = item - nblocks;
      const int4 sg = segs[si];  // partial slot, k_begin, k_end, long-row index
      const int32_t row = long_rows[sg.w];
      if (kFiltered && !flt.keep(row)) continue;
      T acc = sr.neutral();
      for (int32_t base = sg.y; base < sg.z; base += 32 * 4) {
        T v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int32_t k = base + u * 32 + lane;
          v[u] = (k < sg.z) ? sr.mulk(k, __ldcs(colval + k), row + 1) : sr.neutral();
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) acc = sr.addv(acc, v[u]);
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) acc = sr.addv(acc, shfl_xor_m<T>(kFull, acc, off, 32));
      const int32_t f0 = long_first_seg[sg.w], f1 = long_first_seg[sg.w + 1];
      if (f1 - f0 == 1) {  // the whole row in one segment
        if (acc != acc) acc = warp_refold_row(sr, rowptr, colval, row, lane);
        if (lane == 0) sr.write(row, acc);
        continue;
      }
      unsigned prev = 0;
      if (lane == 0) {
        partials[sg.x] = acc;
        __threadfence();
        prev = atomicAdd(long_count + sg.w, 1u);
      }
      prev = __shfl_sync(kFull, prev, 0);
      if (prev == (unsigned)(f1 - f0 - 1)) {  // this warp completed the row
        __threadfence();
        T tot = sr.neutral();
        if (lane == 0) {
          for (int32_t q = f0; q < f1; ++q) tot = sr.addv(tot, __ldcg(partials + q));
          long_count[sg.w] = 0;  // ready for the next launch
        }
        tot = shfl_idx_m<T>(kFull, tot, 0);
        if (tot != tot) tot = warp_refold_row(sr, rowptr, colval, row, lane);
        if (lane == 0) sr.write(row, tot);
      }
    }
  }
}

// ---------------------------------------------------------------------------------
// SELL: one thread per (stored row, chunk of its slice).  Every thread walks at most
// kSellChunk columns with stride C, so hub slices no longer serialise on one thread;
// a row spread over several chunks is combined in chunk order by k_sell_combine.
// ---------------------------------------------------------------------------------
template <class SR>
__global__ void k_sell(SR sr, const int32_t* __restrict__ slice_ptr,
                       const int32_t* __restrict__ colval, const int32_t* __restrict__ perm,
                       int64_t C, int64_t m, const int4* __restrict__ items, int64_t nitems,
                       typename SR::T* partials, int64_t range_lo, int64_t range_hi,
                       const void* mask, int tmask) {
  typedef typename SR::T T;
  const int64_t total = nitems * C;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t it = t / C, o = t - it * C;
    const int4 d = items[it];  // slice, first column, end column, partial index
    const int64_t srow = (int64_t)d.x * C + o;
    if (srow >= m) continue;
    const int64_t r1 = perm ? (int64_t)perm[srow] : srow + 1;  // original row, 1-based
    if (range_lo > 0 && (r1 < range_lo || r1 > range_hi)) continue;
    if (mask && raw_is_zero(load_raw(mask, tmask, r1 - 1), tmask)) continue;
    int64_t i = (int64_t)slice_ptr[d.x] - 1 + o + (int64_t)d.y * C;
    T acc = sr.neutral();
    int32_t j = d.y;
    bool done = false;
    for (; j + 8 <= d.z && !done; j += 8, i += 8 * C) {
      int32_t c[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) c[u] = ld_stream(colval + i + u * C);
      T p[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) p[u] = (c[u] != -1) ? sr.mulk(i + u * C, c[u], r1) : sr.neutral();
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        if (c[u] == -1) { done = true; break; }
        acc = sr.addv(acc, p[u]);
      }
    }
    for (; j < d.z && !done; ++j, i += C) {
      const int32_t col = ld_stream(colval + i);
      if (col == -1) break;
      acc = sr.addv(acc, sr.mulk(i, col, r1));
    }
    if (d.w < 0) sr.write(r1 - 1, acc);
    else partials[(int64_t)d.w * C + o] = acc;
  }
}

// one warp per (multi-chunk slice, row): lanes fold the chunk partials lane-strided,
// then a shuffle tree.  A row of <= kSellChunk entries has one non-neutral partial,
// so its value is unchanged (x + 0 == x; the partials are never -0.0).
template <class SR>
__global__ void k_sell_combine(SR sr, const int32_t* __restrict__ perm, int64_t C, int64_t m,
                               const int4* __restrict__ multi, int64_t nmulti,
                               const typename SR::T* __restrict__ partials, int64_t range_lo,
                               int64_t range_hi, const void* mask, int tmask) {
  typedef typename SR::T T;
  const int lane = threadIdx.x & 31;
  const int64_t total = nmulti * C;
  for (int64_t t = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < total;
       t += ((int64_t)gridDim.x * blockDim.x) >> 5) {
    const int64_t q = t / C, o = t - q * C;
    const int4 d = multi[q];  // slice, first partial, chunks
    const int64_t srow = (int64_t)d.x * C + o;
    if (srow >= m) continue;
    const int64_t r1 = perm ? (int64_t)perm[srow] : srow + 1;
    if (range_lo > 0 && (r1 < range_lo || r1 > range_hi)) continue;
    if (mask && raw_is_zero(load_raw(mask, tmask, r1 - 1), tmask)) continue;
    T acc = sr.neutral();
    for (int32_t c = lane; c < d.z; c += 32) acc = sr.addv(acc, partials[(int64_t)(d.y + c) * C + o]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc = sr.addv(acc, shfl_xor_m<T>(kFull, acc, off, 32));
    if (lane == 0) sr.write(r1 - 1, acc);
  }
}

inline int grid_for(gg_ctx* ctx, int64_t threads, int block) {
  int64_t g = (threads + block - 1) / block;
  int64_t cap = (int64_t)ctx->num_sms * 16;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return (int)g;
}

template <class SR, bool kFiltered, bool kNeedsRow>
int launch_rowblock_t(gg_ctx* ctx, gg_mat* A, const SR& sr, const RowFilter& flt) {
  GG_CHECK(build_row_blocks(ctx, A));
  RowBlocks* rb = A->blocks;
  const int64_t items = rb->nblocks + rb->nsegs;
  if (items == 0) return GG_OK;
  static int per_sm = 0;
  if (per_sm == 0) {
    GG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &per_sm, k_csr_rowblock<SR, kFiltered, kNeedsRow>, kRBWarps * 32, 0));
    if (per_sm < 1) per_sm = 1;
  }
  int64_t grid = (items + kRBWarps - 1) / kRBWarps;
  const int64_t cap = (int64_t)ctx->num_sms * per_sm;  // one resident wave
  if (grid > cap) grid = cap;
  const int tr = trace_main_begin(ctx);
  k_csr_rowblock<SR, kFiltered, kNeedsRow><<<(int)grid, kRBWarps * 32, 0, ctx->stream>>>(
      sr, A->rowptr, A->colval, rb->blocks, rb->nblocks, rb->segs, rb->nsegs, rb->long_first_seg,
      rb->long_rows, rb->long_count, static_cast<typename SR::T*>(rb->partials), flt);
  trace_main_end(ctx, tr);
  trace_count(ctx, 1);
  GG_CUDA(cudaGetLastError());
  return GG_OK;
}

template <class SR>
int launch_rowblock(gg_ctx* ctx, gg_mat* A, const SR& sr, const void* mask = nullptr,
                    int tmask = 0, int64_t lo = 0, int64_t hi = 0, bool needs_row = false) {
  RowFilter flt;
  flt.mask = mask;
  flt.tmask = tmask;
  flt.lo = lo > 0 ? lo - 1 : 0;
  flt.hi = lo > 0 ? hi : A->m;
  const bool filtered = mask != nullptr || lo > 0;
  if (needs_row) {
    if (filtered) return launch_rowblock_t<SR, true, true>(ctx, A, sr, flt);
    return launch_rowblock_t<SR, false, true>(ctx, A, sr, flt);
  }
  if (filtered) return launch_rowblock_t<SR, true, false>(ctx, A, sr, flt);
  return launch_rowblock_t<SR, false, false>(ctx, A, sr, flt);
}

template <class SR>
static int launch_sell(gg_ctx* ctx, gg_mat* A, const SR& sr, const void* mask, int tmask,
                       int64_t lo, int64_t hi, const int32_t* colval_override = nullptr) {
  GG_CHECK(build_sell_plan(ctx, A));
  SellPlan* P = A->sellplan;
  const int64_t C = A->slice_size;
  typedef typename SR::T T;
  if (P->nitems > 0) {
    const int tr = trace_main_begin(ctx);
    k_sell<SR><<<grid_for(ctx, P->nitems * C, 256), 256, 0, ctx->stream>>>(
        sr, A->slice_ptr, colval_override ? colval_override : A->colval,
        A->sigma > 1 ? A->perm : nullptr, C, A->m, P->items,
        P->nitems, static_cast<T*>(P->partials), lo, hi, mask, tmask);
    trace_main_end(ctx, tr);
    trace_count(ctx, 1);
  }
  if (P->nmulti > 0) {
    k_sell_combine<SR><<<grid_for(ctx, P->nmulti * C * 32, 256), 256, 0, ctx->stream>>>(
        sr, A->sigma > 1 ? A->perm : nullptr, C, A->m, P->multi, P->nmulti,
        static_cast<const T*>(P->partials), lo, hi, mask, tmask);
    trace_count(ctx, 1);
  }
  GG_CUDA(cudaGetLastError());
  return GG_OK;
}

}  // namespace gg
