// gg_spmv_typed.cu -- SpMV of the common semirings with operators and element type fixed
// at compile time (gpu_spmv!, src/spmv/CSR.jl and src/spmv/SELL.jl of GPUGraphs.jl).
//
// SRGen reads every value through a (64-bit integer, double) pair and two switches over
// 20 operators, some 60 instructions per entry: R-MAT products ran at 4 to 19% of the
// copy bandwidth.  Matrix, operand and result of one type with (mul, add),
// (add | safe_add, min) on Int32 / Int64 / Float32 / Float64 or (and, or) on Bool take
// SRTyped instead, any accum and mask:
//  * CSR handles of >= kTypedCopyRows rows: the SELL-32 copy with rows sorted by length
//    that the Float32 plus-times product uses, by k_sell32_typed below;
//  * smaller ones, row ranges, and copies that do not fit: the row blocks;
//  * SELL-32 handles: k_sell32_typed on their own arrays; other slice heights: k_sell.
// Rows fold in storage order within chunks of kSellChunk entries, as everywhere.
// Measured, us before -> now: Int32 min-plus R-MAT 21 422 -> 178; masked Bool or-and
// R-MAT 20 307 -> 43; Float64 plus-times R-MAT 20 608 -> 169 (bound by the FP64 pipe: a
// multiply and an add per entry, 100 us), on a SELL-32 handle with sigma 1024 975 -> 152;
// masked Float32 plus-times R-MAT 20 328 -> 81; Int32 min-plus on a 2^20-vertex ER graph
// 102 -> 70 and a 1024 x 1024 grid 28 -> 17.
#include "gg_spmv_kernels.cuh"

namespace gg {

int build_colperm(gg_ctx* ctx, gg_mat* A);  // gg_spmv.cu

// the matrix stream (past L1, evict-first in L2) and the gathered operand (evict-last) of
// any element type, by size
template <typename T>
__device__ __forceinline__ T ld_matrix(const T* p, uint64_t pol) {
  if constexpr (sizeof(T) == 4) {
    int32_t r;
    asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.L2::256B.b32 %0, [%1], %2;" : "=r"(r) : "l"(p), "l"(pol));
    return *reinterpret_cast<T*>(&r);
  } else if constexpr (sizeof(T) == 8) {
    int64_t r;
    asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.L2::256B.b64 %0, [%1], %2;" : "=l"(r) : "l"(p), "l"(pol));
    return *reinterpret_cast<T*>(&r);
  } else {
    int32_t r;
    asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.L2::256B.u8 %0, [%1], %2;" : "=r"(r) : "l"(p), "l"(pol));
    return (T)r;
  }
}
template <typename T>
__device__ __forceinline__ T ld_operand(const T* p, uint64_t pol) {
  if constexpr (sizeof(T) == 4) {
    int32_t r;
    asm volatile("ld.global.nc.L2::cache_hint.b32 %0, [%1], %2;" : "=r"(r) : "l"(p), "l"(pol));
    return *reinterpret_cast<T*>(&r);
  } else if constexpr (sizeof(T) == 8) {
    int64_t r;
    asm volatile("ld.global.nc.L2::cache_hint.b64 %0, [%1], %2;" : "=l"(r) : "l"(p), "l"(pol));
    return *reinterpret_cast<T*>(&r);
  } else {
    int32_t r;
    asm volatile("ld.global.nc.L2::cache_hint.u8 %0, [%1], %2;" : "=r"(r) : "l"(p), "l"(pol));
    return (T)r;
  }
}

// operators of src/algebra.jl on one type (the semantics of apply_op)
template <int OP, typename T>
__device__ __forceinline__ T typed_op(T x, T y) {
  if constexpr (OP == GG_OP_ADD) return w_add(x, y);
  if constexpr (OP == GG_OP_MUL) return w_mul(x, y);
  if constexpr (OP == GG_OP_MIN) return jl_min<T>(x, y);
  if constexpr (OP == GG_OP_BAND) return bit_and<T>(x, y);
  if constexpr (OP == GG_OP_BOR) return bit_or<T>(x, y);
  if constexpr (OP == GG_OP_SAFE_ADD) return safe_add<T>(x, y);
  return x;
}
// Float32 min by the instruction that propagates NaN and orders -0.0 below +0.0 (the
// comparison form is eight instructions; a NaN's bits are set when the row is written)
template <>
__device__ __forceinline__ float typed_op<GG_OP_MIN, float>(float x, float y) {
  float r;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(x), "f"(y));
  return r;
}
// safe_add on floats: x + y, except that +Inf with -Inf is +Inf (a NaN operand stays NaN)
template <>
__device__ __forceinline__ float typed_op<GG_OP_SAFE_ADD, float>(float x, float y) {
  const float s = __fadd_rn(x, y);
  return (s != s && x == x && y == y) ? __int_as_float(0x7f800000) : s;
}
// Float64 compares run on the FP64 pipe (two lanes a clock and SM here): min and the NaN
// tests work on the bits, whose integer order (sign-magnitude folded) is the values' order
// with -0.0 below +0.0.  Min-plus on R-MAT scale 20: 753 us with comparisons, 565 so.
__device__ __forceinline__ bool nan_bits(int64_t b) {
  return (b & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL;
}
template <>
__device__ __forceinline__ double typed_op<GG_OP_SAFE_ADD, double>(double x, double y) {
  const double s = __dadd_rn(x, y);
  if (nan_bits(__double_as_longlong(s)) && !nan_bits(__double_as_longlong(x)) &&
      !nan_bits(__double_as_longlong(y)))
    return __longlong_as_double(0x7ff0000000000000LL);
  return s;
}
template <>
__device__ __forceinline__ double typed_op<GG_OP_MIN, double>(double x, double y) {
  const int64_t a = __double_as_longlong(x), b = __double_as_longlong(y);
  if (nan_bits(a) || nan_bits(b)) return __longlong_as_double(0x7ff8000000000000LL);
  const int64_t ka = a ^ ((a >> 63) & 0x7fffffffffffffffLL), kb = b ^ ((b >> 63) & 0x7fffffffffffffffLL);
  return ka < kb ? x : y;
}

// kStop: the CSR kernel's stop at the absorbing value (src/spmv/CSR.jl:47-52); SELL
// products have none (src/spmv/SELL.jl:54-60)
template <int TC, int MUL, int ADD, bool kStop>
struct SRTyped {
  typedef typename CType<TC>::T T;
  static const bool kHasAbsorbCheck = kStop;
  static const int kType = TC;
  const T* __restrict__ nz;
  const T* __restrict__ x;
  T* y;
  int accum;
  __device__ __forceinline__ static T fix(T v) {
    if constexpr (TC == GG_BOOL) return v != 0;
    return v;
  }
  __device__ __forceinline__ static T absorb() {
    if constexpr (ADD == GG_OP_ADD) return Lim<T>::max();
    if constexpr (ADD == GG_OP_MIN) return Lim<T>::min();
    return all_ones<T>();
  }
  __device__ __forceinline__ T neutral() const {
    if constexpr (ADD == GG_OP_MIN) return Lim<T>::max();
    return T(0);
  }
  __device__ __forceinline__ bool is_absorb(T a) const { return kStop && a == absorb(); }
  __device__ __forceinline__ T mul(T a, T b) const { return typed_op<MUL, T>(fix(a), fix(b)); }
  __device__ __forceinline__ T mulk(int64_t k, int32_t col1, int64_t, int64_t = 0) const {
    return mul(__ldcs(nz + k), __ldg(x + (col1 - 1)));
  }
  __device__ __forceinline__ T addv(T acc, T v) const { return typed_op<ADD, T>(acc, v); }
  // One step of the fold.  Whole sums stop at typemax here; minima of whole numbers and
  // ors keep the absorbing value by themselves; a Float fold that goes on after it differs
  // only by ending NaN, and such a row is folded again with the stop (kRefold: a select per
  // entry cost a third of the Float64 product).
  static const bool kRefold = kStop && TC >= GG_FLOAT32;
  __device__ __forceinline__ T step(T acc, T v) const {
    if constexpr (kStop && ADD == GG_OP_ADD && TC < GG_FLOAT32)
      return acc == absorb() ? acc : addv(acc, v);
    return addv(acc, v);
  }
  __device__ __forceinline__ void write(int64_t row0, T acc) const {
    if constexpr (ADD == GG_OP_MIN && TC == GG_FLOAT32)
      if (acc != acc) acc = __int_as_float(0x7fc00000);
    accum_store_t<TC, TC>(y, row0, acc, accum, row0 + 1, 1, row0 + 1, 1);
  }
};

// ---------------------------------------------------------------------------------
// SELL-32: a warp per work item of the plan (a chunk of <= kSellChunk columns of a slice,
// or a group of narrow slices), lane = row, as k_sell_hot32; the next columns and values
// are loaded while the current operands are gathered.  kHot: the 128 KB of x that the
// most frequent columns gather sit in shared memory (columns relabelled by frequency;
// 32768 values of 4 bytes, 16384 of 8, 131072 Bools), one CTA of 1024 threads an SM;
// otherwise (no skew, or x small) CTAs of 256 threads and the whole L1.
// Bound by the gathers that miss the shared part, as the Float32 product is.
// ---------------------------------------------------------------------------------
static const int kTypedHotBytes = 128 << 10;
static const int kTypedHotThreads = 1024;
// Columns up to which x is gathered as it lies: L2 holds it, and ranking and relabelling the
// columns (0.3 ms of the first product), reordering x and filling the shared part of every
// SM cost more than they save.  With the shared part / without, us, R-MAT scale 16, 18, 20:
// Int32 min-plus 54 / 32, 65 / 44, 106 / 98; Float64 min-plus 261 / 90, 284 / 178, 551 / 442
// (its few full SMs wait for the FP64 pipe); masked or-and 51 / 30, 67 / 34, 81 / 49.  Scale
// 21: Int32 177 / 198.
static const int64_t kTypedHotCols = 1 << 20;

struct TypedFilter {  // rows whose results are wanted (1-based range, 0 = all)
  const void* mask;
  int tmask;
  int64_t lo, hi;
  __device__ __forceinline__ bool keep(int64_t r1) const {
    if (lo > 0 && (r1 < lo || r1 > hi)) return false;
    return !mask || !raw_is_zero(load_raw(mask, tmask, r1 - 1), tmask);
  }
};

template <class SR, bool kHot>
__global__ void __launch_bounds__(kHot ? kTypedHotThreads : 256, kHot ? 1 : 4)
    k_sell32_typed(SR sr, const typename SR::T* __restrict__ x, const int32_t* __restrict__ colval,
                   const int32_t* __restrict__ perm, int64_t m, const int4* __restrict__ pitems,
                   int64_t nitems, typename SR::T* partials, int hot, TypedFilter flt) {
  typedef typename SR::T T;
  constexpr int U = sizeof(T) == 8 ? 4 : 8;  // entries of a row in flight
  // whether a warp looks for an early end: Bool sums end at the first true, a SELL handle's
  // own slices may be padded (a CSR's copy is not: rows of one length share a slice)
  constexpr bool kEarly = SR::kType == GG_BOOL || !SR::kHasAbsorbCheck;
  extern __shared__ __align__(16) unsigned char typed_smem[];
  const T* sx = reinterpret_cast<const T*>(typed_smem);
  if (kHot) {
    T* w = reinterpret_cast<T*>(typed_smem);
    for (int i = threadIdx.x; i < hot; i += blockDim.x) w[i] = __ldg(x + i);
    __syncthreads();
  }
  const uint64_t pol_s = l2_evict_first(), pol_x = l2_evict_last();
  // loads only: products are formed after all of a group's gathers are out (with the
  // product inside the branch the gathers waited for one another)
  auto xat = [&](int32_t col1) -> T {
    T v = T(0);
    if (col1 > 0) v = kHot && col1 <= hot ? sx[col1 - 1] : ld_operand(x + (col1 - 1), pol_x);
    return v;
  };
  const int lane = threadIdx.x & 31;
  const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  int4 dn = gw < nitems ? __ldg(pitems + gw) : make_int4(0, 0, 0, -1);
  for (int64_t it = gw; it < nitems; it += nw) {
    const int4 d = dn;  // first position, first stored row, columns (or -slices), partial
    if (it + nw < nitems) dn = __ldg(pitems + it + nw);
    if (d.z < 0) {
      // group of -d.z narrow slices (widths in 4-bit fields of d.w), <= 8 columns in all;
      // the next slice's row ids are loaded while this one folds
      const int ns = -d.z;
      const uint32_t widths = (uint32_t)d.w;
      int total = 0;
      for (int t = 0; t < ns; ++t) total += (widths >> (4 * t)) & 15u;
      auto row_at = [&](int t) -> int32_t {  // 1-based, 0 past the matrix
        const int64_t srow = (int64_t)d.y + t * 32 + lane;
        return srow < m ? (perm ? __ldg(perm + srow) : (int32_t)(srow + 1)) : 0;
      };
      // a row range: groups outside it are passed over (SELL handles alone: ranges of a CSR
      // take the row blocks, and with the check its scale 22 product took 338 us, not 329)
      if constexpr (!SR::kHasAbsorbCheck) {
        if (flt.lo > 0) {
          bool any = false;
          for (int t = 0; t < ns; ++t) {
            const int32_t r = row_at(t);
            any |= r >= flt.lo && r <= flt.hi;
          }
          if (!__any_sync(kFull, any)) continue;
        }
      }
      int32_t c[kNarrowCols];
      T p[kNarrowCols];
#pragma unroll
      for (int u = 0; u < kNarrowCols; ++u) {
        c[u] = u < total ? ld_matrix(colval + d.x + u * 32 + lane, pol_s) : -1;
        p[u] = u < total ? ld_matrix(sr.nz + d.x + u * 32 + lane, pol_s) : T(0);
      }
      int32_t rn = row_at(0);
      {
        T xv[kNarrowCols];
#pragma unroll
        for (int u = 0; u < kNarrowCols; ++u) xv[u] = xat(c[u]);
#pragma unroll
        for (int u = 0; u < kNarrowCols; ++u) p[u] = c[u] > 0 ? sr.mul(p[u], xv[u]) : sr.neutral();
      }
      int u0 = 0;
      for (int t = 0; t < ns; ++t) {
        const int32_t r1 = rn;
        if (t + 1 < ns) rn = row_at(t + 1);
        const int w = (int)((widths >> (4 * t)) & 15u);
        T acc = sr.neutral();
        for (int q = 0; q < w; ++q) {  // p[0] is the group's next entry: exactly w steps a
          acc = sr.step(acc, p[0]);    // slice, where a predicated step per entry and slice
#pragma unroll                         // would keep the FP64 pipe busy with nothing
          for (int u = 0; u + 1 < kNarrowCols; ++u) p[u] = p[u + 1];
        }
        if (SR::kRefold && acc != acc) {
          acc = sr.neutral();
          for (int q = 0; q < w && !sr.is_absorb(acc); ++q) {
            const int32_t at = d.x + (u0 + q) * 32 + lane;
            if (colval[at] <= 0) break;
            acc = sr.addv(acc, sr.mul(sr.nz[at], xat(colval[at])));
          }
        }
        u0 += w;
        if (r1 > 0 && flt.keep(r1)) sr.write(r1 - 1, acc);
      }
      continue;
    }
    const int64_t srow = (int64_t)d.y + lane;
    int32_t r1 = srow < m ? (perm ? __ldg(perm + srow) : (int32_t)(srow + 1)) : 0;
    const bool keep = r1 > 0 && flt.keep(r1);
    if (!__any_sync(kFull, keep)) continue;
    bool live = keep;
    int32_t pos = d.x + lane;
    T acc = sr.neutral();
    // the loads' predicates are the same for the whole warp (a lane whose row is left out
    // reads its share of lines fetched anyway): lane-wise ones became branches, 250 us
    // against 150 for a half-masked Float32 product on R-MAT scale 21
    int32_t c[U];
    T a[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      c[u] = u < d.z ? ld_matrix(colval + pos + u * 32, pol_s) : -1;
      a[u] = u < d.z ? ld_matrix(sr.nz + pos + u * 32, pol_s) : T(0);
    }
    for (int32_t j = 0; j < d.z; j += U) {
      const int32_t pn = pos + U * 32;
      int32_t cn[U];
      T an[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const bool in = j + U + u < d.z;
        cn[u] = in ? ld_matrix(colval + pn + u * 32, pol_s) : -1;
        an[u] = in ? ld_matrix(sr.nz + pn + u * 32, pol_s) : T(0);
      }
      T xv[U];
#pragma unroll
      for (int u = 0; u < U; ++u) xv[u] = xat(keep ? c[u] : -1);
#pragma unroll
      for (int u = 0; u < U; ++u) acc = sr.step(acc, c[u] > 0 ? sr.mul(a[u], xv[u]) : sr.neutral());
      // a row's padding comes last, and nothing follows the absorbing value
      if (kEarly) {
        if (c[U - 1] <= 0 || sr.is_absorb(acc)) live = false;
        if (!__any_sync(kFull, live)) break;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        c[u] = cn[u];
        a[u] = an[u];
      }
      pos = pn;
    }
    if (!keep) continue;
    if (SR::kRefold && acc != acc) {
      acc = sr.neutral();
      for (int32_t j = 0; j < d.z && !sr.is_absorb(acc); ++j) {
        const int32_t col = colval[d.x + lane + j * 32];
        if (col <= 0) break;
        acc = sr.addv(acc, sr.mul(sr.nz[d.x + lane + j * 32], xat(col)));
      }
    }
    if (d.w < 0) sr.write((int64_t)r1 - 1, acc);
    else partials[(int64_t)d.w * 32 + lane] = acc;
  }
}

// Rows of the slices cut into chunks (lane = row: one line per chunk).  Wide slices: a CTA
// each, four shares a warp and a tree over the 32 shares.  Slices of at most kNarrowChunks:
// a warp each, the chunks' loads in flight together.  Both add in the order of
// k_sell_combine (share l has the chunks c = l mod 32; share l joins l + 16, then l + 8, 4,
// 2, 1).  A CSR row whose chunks end NaN is folded again in storage order with the stop.
template <class SR>
__device__ __forceinline__ typename SR::T tree8(const SR& sr, const typename SR::T (&v)[8]) {
  static_assert(kNarrowChunks == 8, "tree over eight values");
  const typename SR::T a = sr.step(v[0], v[4]), b = sr.step(v[1], v[5]);
  const typename SR::T c = sr.step(v[2], v[6]), d = sr.step(v[3], v[7]);
  return sr.step(sr.step(a, c), sr.step(b, d));
}

template <class SR>
__device__ __forceinline__ void typed_finish(const SR& sr, typename SR::T acc, bool live, int32_t r1,
                                             int lane, const int32_t* __restrict__ rowptr,
                                             const int32_t* __restrict__ colval) {
  unsigned bad = SR::kRefold ? __ballot_sync(kFull, live && acc != acc) : 0u;
  while (bad) {
    const int b = __ffs(bad) - 1;
    bad &= bad - 1;
    const typename SR::T v =
        warp_refold_row(sr, rowptr, colval, (int64_t)__shfl_sync(kFull, r1, b) - 1, lane);
    if (lane == b) acc = v;
  }
  if (live) sr.write((int64_t)r1 - 1, acc);
}

template <class SR>
__global__ void __launch_bounds__(256)
    k_sell32_typed_combine(SR sr, const int32_t* __restrict__ perm, int64_t m,
                           const int4* __restrict__ wide, int64_t nwide,
                           const int4* __restrict__ narrow, int64_t nnarrow,
                           const typename SR::T* __restrict__ partials, TypedFilter flt,
                           const int32_t* __restrict__ rowptr, const int32_t* __restrict__ colval) {
  typedef typename SR::T T;
  __shared__ T part[8][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto row_at = [&](int32_t slice) -> int32_t {  // 1-based, 0: not wanted
    const int64_t srow = (int64_t)slice * 32 + lane;
    if (srow >= m) return 0;
    const int32_t r1 = perm ? __ldg(perm + srow) : (int32_t)(srow + 1);
    return flt.keep(r1) ? r1 : 0;
  };
  const int64_t nblk = nwide + (nnarrow + 7) / 8;
  for (int64_t q = blockIdx.x; q < nblk; q += gridDim.x) {
    if (q >= nwide) {
      const int64_t i = (q - nwide) * 8 + warp;
      if (i >= nnarrow) continue;
      const int4 d = narrow[i];  // slice, first partial, chunks
      T p[kNarrowChunks];
#pragma unroll
      for (int c = 0; c < kNarrowChunks; ++c)
        p[c] = c < d.z ? partials[(int64_t)(d.y + c) * 32 + lane] : sr.neutral();
      const int32_t r1 = row_at(d.x);
      typed_finish(sr, tree8(sr, p), r1 > 0, r1, lane, rowptr, colval);
      continue;
    }
    const int4 d = wide[q];
    const int32_t r1 = row_at(d.x);
    T acc[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) acc[k] = sr.neutral();
    // chunks of a warp in flight (a hub's slice has a thousand and more).  4 / 16, us:
    // or-and scale 20 88.8 / 82.6, min-plus Int32 scale 21 177.6 / 172.9, Float64 scale 20
    // 203.7 / 204.8
    constexpr int kFly = sizeof(T) == 8 ? 4 : 16;
    for (int c = warp; c < d.z; c += 8 * kFly) {
      T v[kFly];
#pragma unroll
      for (int k = 0; k < kFly; ++k)
        v[k] = c + 8 * k < d.z ? partials[(int64_t)(d.y + c + 8 * k) * 32 + lane] : sr.neutral();
#pragma unroll
      for (int k = 0; k < kFly; ++k) acc[k & 3] = sr.step(acc[k & 3], v[k]);
    }
    part[warp][lane] = sr.step(sr.step(acc[0], acc[2]), sr.step(acc[1], acc[3]));
    __syncthreads();
    if (warp == 0) {
      T v[8];
#pragma unroll
      for (int w = 0; w < 8; ++w) v[w] = part[w][lane];
      typed_finish(sr, tree8(sr, v), r1 > 0, r1, lane, rowptr, colval);
    }
    __syncthreads();
  }
}

template <typename T>
__global__ void k_gather_typed(const T* __restrict__ x, const int32_t* __restrict__ inv, int64_t n, T* xr) {
  // four ranks of a thread in flight
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += 4 * stride) {
    int32_t c[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) c[u] = i + u * stride < n ? __ldg(inv + i + u * stride) : 0;
    T v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = __ldg(x + c[u]);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (i + u * stride < n) xr[i + u * stride] = v[u];
  }
}

// S: the SELL-32 arrays; A: the CSR handle they were made of (nullptr for a SELL handle).
// The reordered x and the chunks' partials are the matrix's (calls on one matrix are
// ordered), as for the Float32 plus-times product.
template <class SR>
static int launch_sell32_typed(gg_ctx* ctx, gg_mat* S, const gg_mat* A, SR sr, const TypedFilter& flt) {
  typedef typename SR::T T;
  GG_CHECK(build_sell_plan(ctx, S));
  if (S->n > kTypedHotCols) GG_CHECK(build_colperm(ctx, S));
  const SellPlan* P = S->sellplan;
  const bool hot_x = S->n > kTypedHotCols && S->colperm->enabled;
  const int32_t* colval = hot_x ? S->colperm->colval_r : S->colval;
  const int32_t* perm = S->sigma > 1 ? S->perm : nullptr;
  const T* x = sr.x;  // sr keeps the caller's x for the refolds over A's own columns
  T* partials = static_cast<T*>(P->partials);
  if (hot_x) {
    T* xr = reinterpret_cast<T*>(S->colperm->xr);
    k_gather_typed<T><<<grid_for(ctx, S->n, 256), 256, 0, ctx->stream>>>(sr.x, S->colperm->inv, S->n, xr);
    trace_count(ctx, 1);
    x = xr;
  }
  sr.nz = static_cast<const T*>(S->nzval);
  cudaError_t e = cudaSuccess;
  if (P->npitems > 0) {
    const int tr = trace_main_begin(ctx);
    if (hot_x) {
      const int64_t cap = kTypedHotBytes / (int64_t)sizeof(T);
      const int hot = (int)(S->n < cap ? S->n : cap);
      e = cudaFuncSetAttribute(k_sell32_typed<SR, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               kTypedHotBytes);
      if (e == cudaSuccess)
        k_sell32_typed<SR, true><<<ctx->num_sms, kTypedHotThreads, hot * sizeof(T), ctx->stream>>>(
            sr, x, colval, perm, S->m, P->pitems, P->npitems, partials, hot, flt);
    } else {
      k_sell32_typed<SR, false><<<grid_for(ctx, P->npitems * 32, 256), 256, 0, ctx->stream>>>(
          sr, x, colval, perm, S->m, P->pitems, P->npitems, partials, 0, flt);
    }
    trace_main_end(ctx, tr);
    trace_count(ctx, 1);
  }
  if (P->nmulti > 0 && e == cudaSuccess) {
    if (A) sr.nz = static_cast<const T*>(A->nzval);
    const int64_t cap = (int64_t)ctx->num_sms * 8, nblk = P->nwide + (P->nnarrow + 7) / 8;
    k_sell32_typed_combine<SR><<<(int)(nblk < cap ? nblk : cap), 256, 0, ctx->stream>>>(
        sr, perm, S->m, P->wide, P->nwide, P->narrow, P->nnarrow, partials, flt,
        A ? A->rowptr : nullptr, A ? A->colval : nullptr);
    trace_count(ctx, 1);
  }
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_error(e, "typed SELL product");
  return GG_OK;
}

// CSR handles of at least this many rows run on the SELL-32 copy (the line of the Float32
// plus-times product; the copy costs nnz x (4 + element) bytes and is made once)
static const int64_t kTypedCopyRows = 1 << 16;

template <int TC, int MUL, int ADD>
static int spmv_typed_t(gg_ctx* ctx, gg_mat* A, int accum, void* y, const void* x, const void* mask,
                        int tmask, int64_t lo, int64_t hi) {
  typedef typename CType<TC>::T T;
  const TypedFilter flt{mask, tmask, lo, hi};
  if (A->format == GG_FMT_SELL) {
    const SRTyped<TC, MUL, ADD, false> sr{static_cast<const T*>(A->nzval), static_cast<const T*>(x),
                                          static_cast<T*>(y), accum};
    // (relabelled columns are a layout of their own: not for values that may not last)
    if (A->slice_size == 32 &&
        (A->n <= kTypedHotCols || A->colperm || (A->copy_due() && !(A->values_churn && capturing(ctx)))))
      return launch_sell32_typed(ctx, A, nullptr, sr, flt);
    return launch_sell(ctx, A, sr, mask, tmask, lo, hi);
  }
  const SRTyped<TC, MUL, ADD, true> sr{static_cast<const T*>(A->nzval), static_cast<const T*>(x),
                                       static_cast<T*>(y), accum};
  const bool large = lo == 0 && A->m >= kTypedCopyRows;
  if (large) ++A->products;
  // values that may not last get no copy; one that another product made is taken
  if (large && !A->no_sell_copy &&
      (A->sell_copy || (A->copy_due() && !(A->values_churn && capturing(ctx))))) {
    if (ensure_sell_copy(ctx, A) != GG_OK) {
      A->sell_copy = nullptr;  // no room for the copy, or past its index range: row blocks
      A->no_sell_copy = true;
    }
    if (A->sell_copy && A->sell_copy->slice_size == 32)
      return launch_sell32_typed(ctx, A->sell_copy, A, sr, flt);
  }
  return launch_rowblock(ctx, A, sr, mask, tmask, lo, hi);
}

// y = A x (Float32 plus-times, every row) on the SELL-32 copy that CSR handle A has: made by
// the built-in rule or, at any size, by a tuned choice
int spmv_typed_on_copy(gg_ctx* ctx, gg_mat* A, const float* x, float* y) {
  const SRTyped<GG_FLOAT32, GG_OP_MUL, GG_OP_ADD, true> sr{static_cast<const float*>(A->nzval), x, y,
                                                          GG_OP_SECOND};
  return launch_sell32_typed(ctx, A->sell_copy, A, sr, TypedFilter{nullptr, 0, 0, 0});
}

template <int TC>
static int spmv_typed_num(gg_ctx* ctx, gg_mat* A, int mul, int add, int accum, void* y, const void* x,
                          const void* mask, int tmask, int64_t lo, int64_t hi, bool* done) {
  *done = true;
  if (mul == GG_OP_MUL && add == GG_OP_ADD)
    return spmv_typed_t<TC, GG_OP_MUL, GG_OP_ADD>(ctx, A, accum, y, x, mask, tmask, lo, hi);
  if (mul == GG_OP_ADD && add == GG_OP_MIN)
    return spmv_typed_t<TC, GG_OP_ADD, GG_OP_MIN>(ctx, A, accum, y, x, mask, tmask, lo, hi);
  if (mul == GG_OP_SAFE_ADD && add == GG_OP_MIN)
    return spmv_typed_t<TC, GG_OP_SAFE_ADD, GG_OP_MIN>(ctx, A, accum, y, x, mask, tmask, lo, hi);
  *done = false;
  return GG_OK;
}

// *done: whether the product was one of the fixed semirings (and was run)
int spmv_typed(gg_ctx* ctx, gg_mat* A, int tc, int mul, int add, int accum, void* y, int ty,
               const void* x, int tx, const void* mask, int tmask, int64_t lo, int64_t hi, bool* done) {
  *done = false;
  if (A->dtype != tc || tx != tc || ty != tc) return GG_OK;
  switch (tc) {
    case GG_BOOL:
      if ((mul != GG_OP_BAND && mul != GG_OP_LAND) || (add != GG_OP_BOR && add != GG_OP_LOR)) return GG_OK;
      *done = true;
      return spmv_typed_t<GG_BOOL, GG_OP_BAND, GG_OP_BOR>(ctx, A, accum, y, x, mask, tmask, lo, hi);
    case GG_INT32: return spmv_typed_num<GG_INT32>(ctx, A, mul, add, accum, y, x, mask, tmask, lo, hi, done);
    case GG_INT64: return spmv_typed_num<GG_INT64>(ctx, A, mul, add, accum, y, x, mask, tmask, lo, hi, done);
    case GG_FLOAT32: return spmv_typed_num<GG_FLOAT32>(ctx, A, mul, add, accum, y, x, mask, tmask, lo, hi, done);
    default: return spmv_typed_num<GG_FLOAT64>(ctx, A, mul, add, accum, y, x, mask, tmask, lo, hi, done);
  }
}

}  // namespace gg
