// gg_layout.cu -- orders and fills of the derived layouts, on the device.
//
//  * sort_rows_by_length: the row order of SELL-C-sigma (rows by decreasing length
//    within windows of sigma rows, equal lengths in row order).
//  * sell_fill: a CSR matrix's entries into the slice-column-major SELL arrays.
//  * sell_resorted: a SELL matrix again as SELL-32 with its rows sorted over the whole
//    matrix.
//  * rank_columns: columns by decreasing number of entries (equal counts by column).
//
// The first call on a matrix pays for these.  On the host (std::stable_sort over the
// rows, std::sort over the columns) and with a thread per SELL row, whose hub rows of
// 10^5 entries are one long chain of loads, they were nearly all of a first search's or
// product's time.  Radix sorts are stable, so the orders are the same ones.  First call on
// new matrices: Float32 product on R-MAT scale 22 437 -> 6.2 ms, Int32 shortest paths on
// R-MAT scale 22 324 -> 81 ms.
#include <vector>

#include <cub/device/device_radix_sort.cuh>

#include "gg_semiring.cuh"

namespace gg {

static int grid_of(gg_ctx* ctx, int64_t work) {
  int64_t g = (work + 255) / 256;
  const int64_t cap = (int64_t)ctx->num_sms * 8;
  if (g > cap) g = cap;
  return (int)(g < 1 ? 1 : g);
}

// Temporaries of one layout in one allocation, each part 256-byte aligned, freed with the
// object (after a wait for the kernels that use them).  Stream-ordered allocations, one a
// part, gave their memory back to the system at every wait of the stream and mapped it again:
// 0.2 to 0.3 ms of a layout of a few thousand rows.
struct TempMem {
  static const int kParts = 6;
  size_t off[kParts + 1] = {0};
  char* base = nullptr;
  cudaError_t error = cudaSuccess;
  cudaStream_t st;
  bool ordered;
  TempMem(cudaStream_t stream, size_t a, size_t b, size_t c = 0, size_t d = 0, size_t e = 0, size_t f = 0)
      : st(stream) {
    const size_t bytes[kParts] = {a, b, c, d, e, f};
    for (int i = 0; i < kParts; ++i) off[i + 1] = off[i] + ((bytes[i] + 255) & ~(size_t)255);
    ordered = off[kParts] > ((size_t)1 << 20);
    error = ordered ? cudaMallocAsync((void**)&base, off[kParts], st)
                    : cudaMalloc((void**)&base, off[kParts] > 0 ? off[kParts] : 1);
    if (error != cudaSuccess) {
      base = nullptr;
      (void)cudaGetLastError();
    }
  }
  ~TempMem() {
    if (ordered && base) cudaFreeAsync(base, st);
    else cudaFree(base);
  }
  TempMem(const TempMem&) = delete;
  TempMem& operator=(const TempMem&) = delete;
  template <typename T>
  T* at(int part) const { return base ? reinterpret_cast<T*>(base + off[part]) : nullptr; }
};

__global__ void k_row_max(int64_t m, const int32_t* __restrict__ rowptr, unsigned* out) {
  int32_t mx = 0;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < m;
       r += (int64_t)gridDim.x * blockDim.x)
    mx = max(mx, rowptr[r + 1] - rowptr[r]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0 && mx > 0) atomicMax(out, (unsigned)mx);
}

__global__ void k_row_keys(int64_t m, const int32_t* __restrict__ rowptr, int64_t sigma,
                           int len_bits, int32_t max_len, uint64_t* key, int32_t* row1) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < m;
       r += (int64_t)gridDim.x * blockDim.x) {
    if (key) key[r] = ((uint64_t)(r / sigma) << len_bits) | (uint32_t)(max_len - (rowptr[r + 1] - rowptr[r]));
    row1[r] = (int32_t)(r + 1);
  }
}

static int bits_of(uint64_t v) {  // bits that hold 0 .. v
  int b = 0;
  while (b < 64 && (v >> b) != 0) ++b;
  return b;
}

// perm[i] (device, m entries): the 1-based row at place i
int sort_rows_by_length(gg_ctx* ctx, const int32_t* rowptr, int64_t m, int64_t sigma, int32_t* perm) {
  if (m == 0) return GG_OK;
  if (sigma <= 1) {
    k_row_keys<<<grid_of(ctx, m), 256, 0, ctx->stream>>>(m, rowptr, 1, 0, 0, nullptr, perm);
    GG_CUDA(cudaGetLastError());
    return GG_OK;
  }
  cudaStream_t st = ctx->stream;
  size_t tmp_bytes = 0;
  unsigned h = 0;
  cudaError_t e = cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, (const uint64_t*)nullptr, (uint64_t*)nullptr,
                                                  (const int32_t*)nullptr, (int32_t*)nullptr, m, 0, 64, st);
  TempMem mem(st, 4, m * sizeof(uint64_t), m * sizeof(uint64_t), m * sizeof(int32_t), tmp_bytes);
  if (e == cudaSuccess) e = mem.error;
  unsigned* mx = mem.at<unsigned>(0);
  uint64_t *key = mem.at<uint64_t>(1), *key2 = mem.at<uint64_t>(2);
  int32_t* row = mem.at<int32_t>(3);
  void* tmp = mem.at<char>(4);
  if (e == cudaSuccess) e = cudaMemsetAsync(mx, 0, sizeof(unsigned), st);
  if (e == cudaSuccess) {
    k_row_max<<<grid_of(ctx, m), 256, 0, st>>>(m, rowptr, mx);
    e = cudaMemcpyAsync(&h, mx, sizeof(unsigned), cudaMemcpyDeviceToHost, st);
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  const int len_bits = bits_of(h);
  const int bits = len_bits + bits_of((uint64_t)((m - 1) / sigma));
  if (e == cudaSuccess) {
    k_row_keys<<<grid_of(ctx, m), 256, 0, st>>>(m, rowptr, sigma, len_bits, (int32_t)h, key, row);
    e = cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, key, key2, row, perm, m, 0, bits > 0 ? bits : 1, st);
  }
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);  // before the temporaries go
  if (e != cudaSuccess) return cuda_error(e, "row order");
  return GG_OK;
}

// widest row of every slice (width cleared before): a thread per stored row, one atomic
// per warp where the warp's rows share a slice, so slices of any height are spread
__global__ void k_slice_width(int64_t m, int64_t C, const int32_t* __restrict__ rowptr,
                              const int32_t* __restrict__ perm, int32_t* width) {
  for (int64_t t0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) & ~(int64_t)31; t0 < m;
       t0 += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t = t0 + (threadIdx.x & 31);
    int32_t len = 0;
    if (t < m) {
      const int32_t r = perm[t];
      len = rowptr[r] - rowptr[r - 1];
    }
    if (t0 / C == (t0 + 31) / C) {
      len = __reduce_max_sync(0xffffffffu, len);
      if ((threadIdx.x & 31) == 0 && len > 0) atomicMax(width + t0 / C, len);
    } else if (len > 0) {
      atomicMax(width + t / C, len);
    }
  }
}

int sell_slice_widths(gg_ctx* ctx, const int32_t* rowptr, const int32_t* perm, int64_t m, int64_t C,
                      int64_t ns, int32_t* width) {
  if (ns == 0) return GG_OK;
  GG_CUDA(cudaMemsetAsync(width, 0, ns * sizeof(int32_t), ctx->stream));
  k_slice_width<<<grid_of(ctx, m), 256, 0, ctx->stream>>>(m, C, rowptr, perm, width);
  GG_CUDA(cudaGetLastError());
  return GG_OK;
}

// Entry p of the SELL arrays for every p: consecutive threads take consecutive places
// (coalesced stores; a slice column's 32 loads come from 32 rows whose next entries share
// the fetched sectors), and a hub row's entries are spread over the whole grid.  The
// slice of p is searched from the one of the thread's previous place.
static const int kFillTile = 4096;  // places per block step

// the last of n segments s with ptr[s] - 1 <= p (ptr ascending, 1-based, p inside): searched
// on from the thread's previous segment, usually one of the next few
struct SegmentCursor {
  int64_t s = 0;
  bool first = true;
  __device__ __forceinline__ void seek(const int32_t* __restrict__ ptr, int64_t n, int64_t p) {
    if (!first && (int64_t)ptr[s + 1] - 1 > p) return;
    int64_t lo = first ? 0 : s + 1, hi = n - 1;
    if (!first)
      for (int64_t step = 1; lo + step < n; step *= 2)
        if ((int64_t)ptr[lo + step] - 1 > p) {
          hi = lo + step - 1;
          break;
        }
    while (lo < hi) {
      const int64_t mid = (lo + hi + 1) >> 1;
      if ((int64_t)ptr[mid] - 1 <= p) lo = mid; else hi = mid - 1;
    }
    s = lo;
    first = false;
  }
};

template <typename V>
__global__ void __launch_bounds__(256)
    k_sell_fill(int64_t m, int32_t C, int64_t ns, int64_t nst, const int32_t* __restrict__ rowptr,
                const int32_t* __restrict__ colval, const V* __restrict__ nz,
                const int32_t* __restrict__ perm, const int32_t* __restrict__ slice_ptr,
                int32_t* s_colval, V* s_nz) {
  for (int64_t tile = (int64_t)blockIdx.x * kFillTile; tile < nst; tile += (int64_t)gridDim.x * kFillTile) {
    const int64_t end = tile + kFillTile < nst ? tile + kFillTile : nst;
    SegmentCursor at;
    for (int64_t p = tile + threadIdx.x; p < end; p += blockDim.x) {
      at.seek(slice_ptr, ns, p);
      const int64_t s = at.s;
      const int32_t rel = (int32_t)(p - ((int64_t)slice_ptr[s] - 1));
      const int32_t j = rel / C, o = rel - j * C;
      const int64_t t = s * C + o;
      int32_t c = -1;
      V v = V(0);
      if (t < m) {
        const int32_t r = perm[t];
        const int32_t k = rowptr[r - 1] - 1 + j;
        if (k < rowptr[r] - 1) {
          c = colval[k];
          v = nz[k];
        }
      }
      s_colval[p] = c;
      s_nz[p] = v;
    }
  }
}

template <typename V>
static void launch_fill(gg_ctx* ctx, const gg_mat* csr, gg_mat* S) {
  int64_t g = (S->n_stored + kFillTile - 1) / kFillTile;
  const int64_t cap = (int64_t)ctx->num_sms * 8;
  if (g > cap) g = cap;
  k_sell_fill<V><<<(int)g, 256, 0, ctx->stream>>>(
      S->m, (int32_t)S->slice_size, S->nslices, S->n_stored, csr->rowptr, csr->colval,
      static_cast<const V*>(csr->nzval), S->perm, S->slice_ptr, S->colval, static_cast<V*>(S->nzval));
}

int sell_fill(gg_ctx* ctx, const gg_mat* csr, gg_mat* S) {
  if (S->n_stored == 0) return GG_OK;
  switch (dtype_size(S->dtype)) {
    case 1: launch_fill<uint8_t>(ctx, csr, S); break;
    case 4: launch_fill<uint32_t>(ctx, csr, S); break;
    default: launch_fill<uint64_t>(ctx, csr, S); break;
  }
  GG_CUDA(cudaGetLastError());
  return GG_OK;
}

// entries of original row r of a SELL matrix: the place of its first padding column
// (entries come first), by bisection -- a hub row walked entry by entry is a chain of
// 10^4 loads
__global__ void k_sell_lengths(int64_t m, int32_t C, const int32_t* __restrict__ slice_ptr,
                               const int32_t* __restrict__ colval, const int32_t* __restrict__ iperm,
                               int32_t* len) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < m;
       r += (int64_t)gridDim.x * blockDim.x) {
    const int32_t t = iperm[r], s = t / C, o = t - s * C;
    const int64_t base = (int64_t)slice_ptr[s] - 1 + o;
    int32_t lo = 0, hi = (slice_ptr[s + 1] - slice_ptr[s]) / C;
    while (lo < hi) {
      const int32_t mid = (lo + hi) >> 1;
      if (colval[base + (int64_t)mid * C] != -1) lo = mid + 1; else hi = mid;
    }
    len[r] = lo;
  }
}

// the entries of SELL matrix A (C, perm inverse iperm) at the places of SELL-32 matrix S
template <typename V>
__global__ void __launch_bounds__(256)
    k_sell_refill(int64_t m, int64_t ns, int64_t nst, const int32_t* __restrict__ perm,
                  const int32_t* __restrict__ slice_ptr, int32_t* s_colval, V* s_nz, int32_t C,
                  const int32_t* __restrict__ a_iperm, const int32_t* __restrict__ a_slice_ptr,
                  const int32_t* __restrict__ a_colval, const V* __restrict__ a_nz) {
  // a warp per slice of S, lane = row: the row's place in A is found once
  const int lane = threadIdx.x & 31;
  for (int64_t it = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; it < ns * 8;
       it += ((int64_t)gridDim.x * blockDim.x) >> 5) {
    const int64_t s = it >> 3, part = it & 7;  // 8 warps share a slice's columns
    const int64_t t = s * 32 + lane, base = (int64_t)slice_ptr[s] - 1 + lane;
    const int32_t width = (slice_ptr[s + 1] - slice_ptr[s]) / 32;
    int64_t from = 0;
    int32_t wide = 0;
    if (t < m) {
      const int32_t at = a_iperm[perm[t] - 1], as = at / C;
      from = (int64_t)a_slice_ptr[as] - 1 + (at - as * C);
      wide = (a_slice_ptr[as + 1] - a_slice_ptr[as]) / C;
    }
#pragma unroll 4
    for (int32_t j = (int32_t)part; j < width; j += 8) {
      int32_t c = -1;
      V v = V(0);
      if (j < wide) {
        c = a_colval[from + (int64_t)j * C];
        v = a_nz[from + (int64_t)j * C];
      }
      s_colval[base + (int64_t)j * 32] = c;
      s_nz[base + (int64_t)j * 32] = v;
    }
  }
}

template <typename V>
static void launch_refill(gg_ctx* ctx, const gg_mat* A, gg_mat* S) {
  k_sell_refill<V><<<grid_of(ctx, S->nslices * 256), 256, 0, ctx->stream>>>(
      S->m, S->nslices, S->n_stored, S->perm, S->slice_ptr, S->colval, static_cast<V*>(S->nzval),
      (int32_t)A->slice_size, A->iperm, A->slice_ptr, A->colval, static_cast<const V*>(A->nzval));
}

// SELL-32 copy of SELL matrix A with rows sorted by length over the whole matrix
int sell_resorted(gg_ctx* ctx, const gg_mat* A, gg_mat** out) {
  *out = nullptr;
  const int64_t m = A->m, ns = (m + 31) / 32;
  const int esz = dtype_size(A->dtype);
  cudaStream_t st = ctx->stream;
  gg_mat* S = new gg_mat();
  S->format = GG_FMT_SELL;
  S->m = m;
  S->n = A->n;
  S->nnz = A->nnz;
  S->dtype = A->dtype;
  S->device = ctx->device;
  S->slice_size = 32;
  S->nslices = ns;
  S->sigma = m;
  TempMem mem(st, m * sizeof(int32_t), (m + 1) * sizeof(int32_t), ns * sizeof(int32_t));
  int32_t *len = mem.at<int32_t>(0), *rp = mem.at<int32_t>(1), *width = mem.at<int32_t>(2);
  std::vector<int32_t> w(ns), sp(ns + 1);
  cudaError_t e = mem.error;
  if (e == cudaSuccess) e = cudaMalloc((void**)&S->perm, m * sizeof(int32_t));
  if (e == cudaSuccess) e = cudaMalloc((void**)&S->slice_ptr, (ns + 1) * sizeof(int32_t));
  int rc = GG_OK;
  if (e == cudaSuccess) {
    k_sell_lengths<<<grid_of(ctx, m), 256, 0, st>>>(m, (int32_t)A->slice_size, A->slice_ptr, A->colval,
                                                    A->iperm, len);
    rc = scan_counts(ctx, len, m, rp, 1);
    if (rc == GG_OK) rc = sort_rows_by_length(ctx, rp, m, m, S->perm);
    if (rc == GG_OK) rc = sell_slice_widths(ctx, rp, S->perm, m, 32, ns, width);
    if (rc == GG_OK) e = cudaMemcpyAsync(w.data(), width, ns * sizeof(int32_t), cudaMemcpyDeviceToHost, st);
    if (rc == GG_OK && e == cudaSuccess) e = cudaStreamSynchronize(st);
  }
  int64_t acc = 1;
  sp[0] = 1;
  for (int64_t s = 0; s < ns && rc == GG_OK && e == cudaSuccess; ++s) {
    acc += (int64_t)w[s] * 32;
    if (acc > (int64_t)INT32_MAX - 4096) rc = set_error(GG_ERR_ARGUMENT, "SELL n_stored exceeds the Int32 index range");
    sp[s + 1] = (int32_t)acc;
  }
  S->n_stored = acc - 1;
  const int64_t nst = S->n_stored > 0 ? S->n_stored : 1;
  if (rc == GG_OK && e == cudaSuccess) e = cudaMalloc((void**)&S->colval, nst * sizeof(int32_t));
  if (rc == GG_OK && e == cudaSuccess) e = cudaMalloc(&S->nzval, nst * esz);
  if (rc == GG_OK && e == cudaSuccess)
    e = cudaMemcpyAsync(S->slice_ptr, sp.data(), (ns + 1) * sizeof(int32_t), cudaMemcpyHostToDevice, st);
  if (rc == GG_OK && e == cudaSuccess) {
    switch (esz) {
      case 1: launch_refill<uint8_t>(ctx, A, S); break;
      case 4: launch_refill<uint32_t>(ctx, A, S); break;
      default: launch_refill<uint64_t>(ctx, A, S); break;
    }
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  }
  if (rc == GG_OK && e != cudaSuccess) rc = cuda_error(e, "sorted SELL copy");
  if (rc != GG_OK) {
    gg_mat_destroy(S);
    return rc;
  }
  *out = S;
  return GG_OK;
}

// ---------------------------------------------------------------------------------
// a CSR matrix's entries by ascending value within each row
// ---------------------------------------------------------------------------------
// ordering bits of a non-negative value: -0.0 (which counts as non-negative, and adds as
// +0.0 does) becomes +0.0
__device__ __forceinline__ uint32_t value_key(uint8_t v) { return v; }
__device__ __forceinline__ uint32_t value_key(uint32_t v) { return v == 0x80000000u ? 0u : v; }

template <typename V>
__global__ void k_value_max(const V* __restrict__ nz, int64_t nnz, unsigned* out) {
  uint32_t mx = 0;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < nnz;
       k += (int64_t)gridDim.x * blockDim.x)
    mx = max(mx, value_key(nz[k]));
  mx = __reduce_max_sync(0xffffffffu, mx);
  if ((threadIdx.x & 31) == 0 && mx) atomicMax(out, mx);
}

template <typename V>
__global__ void __launch_bounds__(256)
    k_entry_keys(int64_t m, int64_t nnz, const int32_t* __restrict__ rowptr, const V* __restrict__ nz,
                 int vbits, uint64_t* __restrict__ key) {
  for (int64_t tile = (int64_t)blockIdx.x * kFillTile; tile < nnz; tile += (int64_t)gridDim.x * kFillTile) {
    const int64_t end = tile + kFillTile < nnz ? tile + kFillTile : nnz;
    SegmentCursor at;
    for (int64_t p = tile + threadIdx.x; p < end; p += blockDim.x) {
      at.seek(rowptr, m, p);
      key[p] = ((uint64_t)at.s << vbits) | value_key(nz[p]);
    }
  }
}

template <typename V>
__global__ void k_key_values(const uint64_t* __restrict__ key, int64_t nnz, int vbits, V* __restrict__ nz) {
  const uint64_t low = (1ull << vbits) - 1;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < nnz;
       k += (int64_t)gridDim.x * blockDim.x)
    nz[k] = (V)(key[k] & low);
}

template <typename V>
static int sort_entries_t(gg_ctx* ctx, const gg_mat* A, int32_t* col, V* nz) {
  const int64_t m = A->m, nnz = A->nnz;
  cudaStream_t st = ctx->stream;
  const V* src = static_cast<const V*>(A->nzval);
  unsigned h = 0;
  size_t tmp_bytes = 0;
  cudaError_t e = cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, (const uint64_t*)nullptr, (uint64_t*)nullptr,
                                                  (const int32_t*)nullptr, (int32_t*)nullptr, nnz, 0, 64, st);
  TempMem mem(st, nnz * sizeof(uint64_t), nnz * sizeof(uint64_t), tmp_bytes);
  if (e == cudaSuccess) e = mem.error;
  uint64_t *key = mem.at<uint64_t>(0), *key2 = mem.at<uint64_t>(1);
  void* tmp = mem.at<char>(2);
  if (e == cudaSuccess) e = cudaMemsetAsync(ctx->d_flags, 0, sizeof(unsigned), st);
  if (e == cudaSuccess) {
    k_value_max<V><<<grid_of(ctx, nnz), 256, 0, st>>>(src, nnz, ctx->d_flags);
    e = cudaMemcpyAsync(ctx->h_flags, ctx->d_flags, sizeof(unsigned), cudaMemcpyDeviceToHost, st);
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  h = ctx->h_flags[0];
  const int vbits = bits_of(h), bits = vbits + bits_of((uint64_t)(m > 0 ? m - 1 : 0));
  if (e == cudaSuccess) {
    int64_t g = (nnz + kFillTile - 1) / kFillTile;
    if (g > (int64_t)ctx->num_sms * 8) g = (int64_t)ctx->num_sms * 8;
    k_entry_keys<V><<<(int)g, 256, 0, st>>>(m, nnz, A->rowptr, src, vbits, key);
    e = cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, key, key2, A->colval, col, nnz, 0,
                                        bits > 0 ? bits : 1, st);
  }
  if (e == cudaSuccess) {
    k_key_values<V><<<grid_of(ctx, nnz), 256, 0, st>>>(key2, nnz, vbits, nz);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return cuda_error(e, "entry order");
  return GG_OK;
}

// A CSR handle's entries ordered by value within each row (values non-negative, 1 or 4
// bytes: their bits order as they do) into col / nz (device, nnz each); rowptr as A's
int sort_entries_by_value(gg_ctx* ctx, const gg_mat* A, int32_t* col, void* nz) {
  if (A->nnz == 0) return GG_OK;
  if (dtype_size(A->dtype) == 1) return sort_entries_t<uint8_t>(ctx, A, col, static_cast<uint8_t*>(nz));
  return sort_entries_t<uint32_t>(ctx, A, col, static_cast<uint32_t*>(nz));
}

__global__ void k_iota(int32_t* p, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    p[i] = (int32_t)i;
}

// rank[inv[i]] = i, and the entries held by the first `top` ranks into *sum
__global__ void k_rank_scatter(int64_t n, const int32_t* __restrict__ inv,
                               const uint32_t* __restrict__ sorted, int64_t top, int32_t* rank,
                               unsigned long long* sum) {
  unsigned long long s = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    rank[inv[i]] = (int32_t)i;
    if (i < top) s += sorted[i];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0 && s) atomicAdd(sum, s);
}

// cnt[c] (device): entries of column c.  inv[i]: the column of rank i (most entries
// first, equal counts by column), rank: its inverse, both n device words; *top_sum: the
// entries of the first `top` ranks.  Synchronises the stream.
int rank_columns(gg_ctx* ctx, const int32_t* cnt, int64_t n, int64_t top, int32_t* inv,
                 int32_t* rank, int64_t* top_sum) {
  size_t tmp_bytes = 0;
  unsigned long long h = 0;
  cudaStream_t st = ctx->stream;
  const uint32_t* key = reinterpret_cast<const uint32_t*>(cnt);
  cudaError_t e = cub::DeviceRadixSort::SortPairsDescending(nullptr, tmp_bytes, (const uint32_t*)nullptr,
                                                            (uint32_t*)nullptr, (const int32_t*)nullptr,
                                                            (int32_t*)nullptr, n, 0, 32, st);
  TempMem mem(st, sizeof(unsigned long long), n * sizeof(uint32_t), n * sizeof(int32_t), tmp_bytes);
  if (e == cudaSuccess) e = mem.error;
  unsigned long long* sum = mem.at<unsigned long long>(0);
  uint32_t* sorted = mem.at<uint32_t>(1);
  int32_t* id = mem.at<int32_t>(2);
  void* tmp = mem.at<char>(3);
  if (e == cudaSuccess) e = cudaMemsetAsync(sum, 0, sizeof(*sum), st);
  if (e == cudaSuccess) {
    k_iota<<<grid_of(ctx, n), 256, 0, st>>>(id, n);
    e = cub::DeviceRadixSort::SortPairsDescending(tmp, tmp_bytes, key, sorted, id, inv, n, 0, 32, st);
  }
  if (e == cudaSuccess) {
    k_rank_scatter<<<grid_of(ctx, n), 256, 0, st>>>(n, inv, sorted, top, rank, sum);
    e = cudaMemcpyAsync(&h, sum, sizeof(h), cudaMemcpyDeviceToHost, st);
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return cuda_error(e, "column ranks");
  *top_sum = (int64_t)h;
  return GG_OK;
}

}  // namespace gg
