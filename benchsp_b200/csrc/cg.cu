// Conjugate gradients on the device: plain FP64 CG and mixed-precision CG
// with reliable updates.  The reference has no solver (the CG /
// mixed-precision rows are absent there); this is the precision form of the
// benchmark's CG configuration: 3-D 7-point Poisson, tolerance 1e-10 on
// ||b - A x|| / ||b|| checked in FP64.
//
// Mixed precision: the matrix is stored a second time, in SELL-32 layout
// (slices of 32 consecutive rows padded to the slice's longest row; entry k of
// the slice's row l at slice_off + 32 k + l, so the 32 rows of a warp read
// each k with one coalesced access), with values in FP32, FP16 or BF16.
// FP16/BF16 values carry one power-of-two exponent per row (v = stored * 2^e,
// the row's largest magnitude scaled into [1, 2); the row sum is scaled once),
// and column indices are stored as int16 offsets from the row
// when every |col - row| < 32768 (banded matrices), else int32.  FP16/BF16
// values with int16 offsets are packed into one 32-bit word per entry.  A
// nonzero then moves 4 bytes instead of 12 (FP64 + int32).  CG iterations
// run on that matrix with FP32 vectors (dot products in FP64).
// The FP64 state is the solution x64 and the true residual: whenever the
// iterated residual has dropped by `reliable_delta` since the last update,
// x64 += x32, r = b - A x64 is recomputed in FP64 with the FP64 matrix and
// replaces the iterated residual, and the search direction is kept (CG with
// reliable updates), so the iteration count stays close to plain FP64 CG while
// most bytes move at low precision.
//
// One CG iteration is two kernels (matrices of few diagonals whose vectors fit
// the SMs' shared memory run a fused form instead, cg_fused_kernel):
//   A. beta = rr_k / rr_{k-1}; p_k = r_k + beta p_{k-1} formed on the fly for
//      every gathered column (r and p_{k-1} are read, p_k written for the own
//      row into the other p buffer); q = A p_k; partials of p_k.q;
//   B. alpha = rr_k / p.q; x += alpha p_k; r -= alpha q; partials of r.r.
// Every CTA reduces the previous kernel's per-CTA partials in the same order
// (deterministic, no atomics).  Scalars ping-pong between two slots by
// iteration parity so no CTA reads a value written in its own launch.  Zero
// denominators freeze the iteration (alpha = beta = 0), so iterations run
// after convergence inside a captured graph are harmless.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <type_traits>
#include <vector>

#include "bsp_internal.cuh"
#include "util.cuh"

namespace bsp {

constexpr int kCgThreads = 256;
constexpr int kRowFirst = 8;  // row entries loaded together per lane

template <typename V> __device__ __forceinline__ float lp_to_float(V v);
template <> __device__ __forceinline__ float lp_to_float<float>(float v) { return v; }
template <> __device__ __forceinline__ float lp_to_float<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float lp_to_float<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

// 2^e as a float built from its exponent bits (|e| <= 126).
__device__ __forceinline__ float pow2f(int e) { return __int_as_float((127 + e) << 23); }

// Deterministic block sum of one double per thread (fixed shuffle tree, then
// the warp totals in order).  Valid in thread 0.
__device__ __forceinline__ double block_sum(double v, double *smem /* [kCgThreads/32] */) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) smem[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < kCgThreads / 32; ++w) t += smem[w];
  __syncthreads();
  return t;
}

// Sum of n partials in index order; every CTA gets the same value.
__device__ __forceinline__ double reduce_partials(const double *__restrict__ part, int n, double *smem) {
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += kCgThreads) s += __ldcg(part + i);
  s = block_sum(s, smem);
  __shared__ double bcast;
  if (threadIdx.x == 0) bcast = s;
  __syncthreads();
  return bcast;
}

// Matrix access: values V with optional group exponents, columns int32 or
// int16 offsets from the row.
// kPacked (FP16/BF16 values with int16 offsets): one 32-bit word per entry,
// value bits low, offset high, so one load gives both.
template <typename V, typename VT, bool SCALED, bool DELTA16>
struct CgMat {
  static constexpr bool kPacked = SCALED && DELTA16 && sizeof(V) == 2;
  const int32_t *rowPtr;  // CSR row pointers (FP64 mode)
  const void *cols;
  const V *val;           // SELL values, or the packed words when kPacked
  const int8_t *exps;
  const int32_t *slice_len;  // SELL-32 (mixed modes)
  const int64_t *slice_off;
  int32_t uniform_len;       // > 0: every slice has this length, offsets are sl * 32 * uniform_len
  __device__ __forceinline__ int64_t col(int64_t r, int32_t j) const {
    if (DELTA16) return r + (int64_t) reinterpret_cast<const int16_t *>(cols)[j];
    return reinterpret_cast<const int32_t *>(cols)[j];
  }
  __device__ __forceinline__ VT value(int32_t j) const { return (VT)val[j]; }  // CSR (FP64) path
};

// Kernel A: p_k = r + beta p_prev (own row stored, gathered columns formed on
// the fly), q = A p_k, partials of p_k.q.  rr_part = partials of rr_k;
// rr_prev_slot = rr_{k-1}; rr_slot receives rr_k (written by CTA 0).
// LPR (FP64 CSR path only): lanes per row; rows longer than ~10 entries
// get 2, 4 or 8 lanes that split the row's entries (4 loads in flight each)
// and combine by shuffle, instead of one thread walking the row.
// The FP64 CSR path fits 40 registers without spills: 6 resident CTAs per SM
// instead of 4 (Poisson 128^3 FP64 CG 37.0 -> 35.9 ms); so does the FP32
// SELL form with 32-bit columns (its default since the uniform-slice field).
// The other SELL forms keep the default (the same cap cost them 15%).
template <typename V, typename VT, bool SCALED, bool DELTA16, int LPR = 1>
__global__ void __launch_bounds__(kCgThreads, (sizeof(V) == 8 || (sizeof(V) == 4 && !DELTA16)) ? 6 : 0)
    cg_dir_spmv_kernel(int32_t n, CgMat<V, VT, SCALED, DELTA16> A,
                                                                 const VT *__restrict__ r,
                                                                 const VT *__restrict__ p_prev,
                                                                 VT *__restrict__ p, VT *__restrict__ q,
                                                                 const double *__restrict__ rr_part, int npart,
                                                                 const double *__restrict__ rr_prev_slot,
                                                                 double *__restrict__ rr_slot,
                                                                 double *__restrict__ pq_part) {
  __shared__ double smem[kCgThreads / 32];
  const double rr = reduce_partials(rr_part, npart, smem);
  const double rr_prev = *rr_prev_slot;
  const double beta = (rr_prev != 0.0 && isfinite(rr)) ? rr / rr_prev : 0.0;
  const VT bt = (VT)beta;
  double dot = 0.0;
  const int64_t stride = (int64_t)gridDim.x * kCgThreads;
  if constexpr (sizeof(V) < 8 || DELTA16) {
    // SELL-32: warp = slice (the grid stride is a multiple of 32 rows); the
    // row's power-of-two scale is applied once to its sum; offsets are 32-bit
    // (the padded matrix has < 2^31 entries).  FP64 values (V = double, 16-bit
    // column offsets) are loaded and multiplied in FP64.
    using Mat = CgMat<V, VT, SCALED, DELTA16>;
    using AV = typename std::conditional<sizeof(V) == 8, double, float>::type;
    const int lane = threadIdx.x & 31;
    for (int64_t i = (int64_t)blockIdx.x * kCgThreads + threadIdx.x; i - lane < n; i += stride) {
      const int32_t sl = (int32_t)(i >> 5);
      // uniform slices (16-bit offset forms; the 32-bit column form would
      // need 8 more registers): length and offset without loads
      const bool uni = DELTA16 && A.uniform_len > 0;
      const int32_t len = uni ? A.uniform_len : A.slice_len[sl];
      const uint32_t base = uni ? (uint32_t)sl * 32u * (uint32_t)A.uniform_len : (uint32_t)A.slice_off[sl];
      const uint32_t off = base + lane;
      const bool live = i < n;
      const int32_t row = (int32_t)i;
      VT acc = VT(0);
      const float row_scale = (SCALED && live) ? pow2f(A.exps[i]) : 1.f;
      {
        const int32_t kb = 0, kn = len;
        for (int32_t k0 = 0; k0 < kn; k0 += kRowFirst) {
          int32_t c[kRowFirst];
          AV a[kRowFirst];
#pragma unroll
          for (int k = 0; k < kRowFirst; ++k) {
            c[k] = row;
            a[k] = AV(0);
            if (k0 + k < kn) {
              const uint32_t j = off + (uint32_t)(kb + k0 + k) * 32u;
              if constexpr (Mat::kPacked) {
                const uint32_t w = __ldg(reinterpret_cast<const uint32_t *>(A.val) + j);
                const unsigned short vb = (unsigned short)(w & 0xffffu);
                if constexpr (std::is_same<V, __half>::value)
                  a[k] = __half2float(__ushort_as_half(vb));
                else
                  a[k] = __bfloat162float(__ushort_as_bfloat16(vb));
                c[k] = row + (int32_t)(int16_t)(w >> 16);
              } else {
                if constexpr (sizeof(V) == 8)
                  a[k] = __ldg(A.val + j);
                else
                  a[k] = lp_to_float<V>(__ldg(A.val + j));
                if (DELTA16)
                  c[k] = row + (int32_t)__ldg(reinterpret_cast<const int16_t *>(A.cols) + j);
                else
                  c[k] = __ldg(reinterpret_cast<const int32_t *>(A.cols) + j);
              }
            }
          }
#pragma unroll
          for (int k = 0; k < kRowFirst; ++k)
            if (k0 + k < kn && live) acc = fma((VT)a[k], fma(bt, __ldg(p_prev + c[k]), __ldg(r + c[k])), acc);
        }
      }
      if constexpr (SCALED) acc *= row_scale;
      if (live) {
        const VT pi = fma(bt, p_prev[i], r[i]);
        p[i] = pi;
        q[i] = acc;
        dot += (double)acc * (double)pi;
      }
    }
  } else if constexpr (LPR > 1) {
    // warp-uniform loop: each pass covers 32 / LPR consecutive rows per warp
    const int lane = threadIdx.x & 31, sub = lane & (LPR - 1);
    const int64_t rstride = stride / LPR;
    for (int64_t base = ((int64_t)blockIdx.x * kCgThreads + (threadIdx.x & ~31)) / LPR; base < n; base += rstride) {
      const int64_t i = base + lane / LPR;
      const bool live = i < n;
      VT acc = VT(0);
      if (live) {
        const int32_t e = A.rowPtr[i + 1];
        int32_t j = A.rowPtr[i] + sub;
        for (; j + 3 * LPR < e; j += 4 * LPR) {
          int64_t c[4];
          VT a[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            c[k] = A.col(i, j + k * LPR);
            a[k] = A.value(j + k * LPR);
          }
#pragma unroll
          for (int k = 0; k < 4; ++k) acc = fma(a[k], fma(bt, __ldg(p_prev + c[k]), __ldg(r + c[k])), acc);
        }
        for (; j < e; j += LPR) {
          const int64_t cj = A.col(i, j);
          acc = fma(A.value(j), fma(bt, __ldg(p_prev + cj), __ldg(r + cj)), acc);
        }
      }
#pragma unroll
      for (int o = LPR / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (live && sub == 0) {
        const VT pi = fma(bt, p_prev[i], r[i]);
        p[i] = pi;
        q[i] = acc;
        dot += (double)acc * (double)pi;
      }
    }
  } else
  for (int64_t i = (int64_t)blockIdx.x * kCgThreads + threadIdx.x; i < n; i += stride) {
    const int32_t s = A.rowPtr[i], e = A.rowPtr[i + 1];
    int64_t c[kRowFirst];
    VT a[kRowFirst];
#pragma unroll
    for (int k = 0; k < kRowFirst; ++k) {
      const int32_t j = s + k;
      c[k] = j < e ? A.col(i, j) : -1;
      a[k] = j < e ? A.value(j) : VT(0);
    }
    VT acc = VT(0);
#pragma unroll
    for (int k = 0; k < kRowFirst; ++k)
      if (c[k] >= 0) acc = fma(a[k], fma(bt, __ldg(p_prev + c[k]), __ldg(r + c[k])), acc);
    for (int32_t j = s + kRowFirst; j < e; ++j) {
      const int64_t cj = A.col(i, j);
      acc = fma(A.value(j), fma(bt, __ldg(p_prev + cj), __ldg(r + cj)), acc);
    }
    const VT pi = fma(bt, p_prev[i], r[i]);
    p[i] = pi;
    q[i] = acc;
    dot += (double)acc * (double)pi;
  }
  const double t = block_sum(dot, smem);
  if (threadIdx.x == 0) {
    pq_part[blockIdx.x] = t;
    if (blockIdx.x == 0) *rr_slot = rr;
  }
}

template <typename V>
__device__ __forceinline__ V from_float_lp(float f);
template <> __device__ __forceinline__ float from_float_lp<float>(float f) { return f; }
template <> __device__ __forceinline__ __half from_float_lp<__half>(float f) { return __float2half_rn(f); }
template <> __device__ __forceinline__ __nv_bfloat16 from_float_lp<__nv_bfloat16>(float f) { return __float2bfloat16_rn(f); }

// ---------------------------------------------------------------------------
// 16-byte vectors of the iteration precision.
template <typename VT> struct Vec16;
template <> struct Vec16<float> { using T = float4; static constexpr int W = 4; };
template <> struct Vec16<double> { using T = double2; static constexpr int W = 2; };

__device__ __forceinline__ float vget(const float4 &v, int k) { return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w; }
__device__ __forceinline__ double vget(const double2 &v, int k) { return k == 0 ? v.x : v.y; }
__device__ __forceinline__ void vset(float4 &v, int k, float a) {
  if (k == 0) v.x = a; else if (k == 1) v.y = a; else if (k == 2) v.z = a; else v.w = a;
}
__device__ __forceinline__ void vset(double2 &v, int k, double a) {
  if (k == 0) v.x = a; else v.y = a;
}

// ---------------------------------------------------------------------------
// Fused iteration: all iterations of a chunk in one cooperative launch, one CTA
// per SM, for matrices of at most kFusedDiags distinct diagonals (grid stencils)
// whose vectors fit in the SMs' shared memory: x, r, p and q of a CTA's rows, 16
// bytes per row in FP32, 32 in FP64.
//
// The two-kernel iteration moves x, r, p and q through L2 several times, gathers
// both r and p_{k-1} for every entry, and pays two launches with a reduction of
// the previous kernel's partials at the head of each.  Here a CTA keeps its
// consecutive slices' rows in shared memory and an iteration is
//   p = r + beta p, published
//   q = A p, p.q                        | grid sum
//   x += alpha p, r -= alpha q, r.r     | grid sum
// with the matrix stored by diagonals (values only, a row's eight in one place)
// and p gathered from shared memory (a column among the CTA's own rows) or from
// the published copy in global memory.  An element is published together with
// the iteration's tag as one word, and a reader loads it again until the tag is
// there: no barrier stands between publishing and gathering.  Every element sees
// the same operations in the same order as in the two kernels (a diagonal that a
// row lacks adds 0 * p); only the dot products' FP64 summation order differs.
//
// A grid sum: each CTA stores {partial, epoch} as one 16-byte word in its slot,
// a thread of every CTA polls each slot until it carries the epoch, and the
// partials are added in a fixed order.  Slots stand 128 bytes apart (side by
// side, stores queue behind the polls of their line: 4.1 against 1.6 us per sum
// with 148 CTAs) and alternate between two arrays: a slot is stored again two
// sums later, when every CTA has read it.  What a CTA read before a sum went
// into its partial, so the published elements need no fence either.
//
// Measured per iteration, Poisson 128^3 FP16 (FP32): two kernels 39 (42) us, here
// 19.7 (20.9): p 2.1, q 11.3, sums 2.9 and 2.9, x and r 1.6.  Everything is in L2
// and shared memory (no DRAM traffic); the product is bound by instruction issue
// and by the 2 of 7 columns that come from another SM.  An earlier form on the
// SELL copy with 16-bit offsets took 31 us (a decode, an address and a test per
// entry).  Whole solves, checks and FP64 residuals included, per iteration: FP64 100^3
// 31.0 -> 22.7 us, FP16 100^3 21.9 -> 15.5, 64^3 11.7 -> 10.3, 24^3 9.0 -> 7.9.  Below
// about 40^3 the two sums are most of an iteration (two_kernels_faster).
//
// The cooperative launch makes all CTAs resident; every wait is bounded all the
// same: kFusedPolls, or in an instantiation of its own (LIMITED) the plan's limit, which
// as an argument of every launch cost registers (FP16 12.34 -> 12.73 ms a solve).  Then
// *err is set and every CTA returns; fused_reset makes the plan usable again.
constexpr int kFusedDiags = 8;
constexpr int kFusedMaxCtas = 256;
constexpr uint32_t kFusedPolls = 1u << 23;  // about 5 s
struct __align__(128) CgSlot {
  double v;
  unsigned long long epoch;
};

// A published element: the value and a tag in one word.
template <typename VT> struct FusedPub;
template <> struct FusedPub<float> {
  using T = unsigned long long;
  static __device__ __forceinline__ T word(float v, uint32_t tag) {
    return (T)tag << 32 | __float_as_uint(v);
  }
  // Column c (relative to the CTA's rows, `mine` of them): *near, or w = *far for a
  // column of another CTA (row0 + c < n).
  static __device__ __forceinline__ void gather(uint32_t c, uint32_t mine, uint32_t row, uint32_t n, uint32_t near,
                                                const T *far, float &v, T &w) {
    asm volatile(
        "{.reg .pred o, f; setp.ge.u32 o, %2, %3; setp.lt.and.u32 f, %4, %5, o;"
        " @!o ld.shared.f32 %0, [%6]; @f ld.relaxed.gpu.global.u64 %1, [%7];}"
        : "+f"(v), "+l"(w)
        : "r"(c), "r"(mine), "r"(row), "r"(n), "r"(near), "l"(far)
        : "memory");
  }
  static __device__ __forceinline__ T get(const T *p) {
    T t;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(t) : "l"(p) : "memory");
    return t;
  }
  static __device__ __forceinline__ void put(T *p, float v, uint32_t tag) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(word(v, tag)) : "memory");
  }
  static __device__ __forceinline__ uint32_t tag(T t) { return (uint32_t)(t >> 32); }
  static __device__ __forceinline__ float value(T t) { return __uint_as_float((uint32_t)t); }
};
struct FusedWord16 {
  unsigned long long lo, hi;
};
__device__ __forceinline__ void st_word16(void *p, unsigned long long lo, unsigned long long hi) {
  asm volatile("{.reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t;}" ::"l"(p), "l"(lo), "l"(hi)
               : "memory");
}
__device__ __forceinline__ FusedWord16 ld_word16(const void *p) {
  FusedWord16 t;
  asm volatile("{.reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t;}"
               : "=l"(t.lo), "=l"(t.hi)
               : "l"(p)
               : "memory");
  return t;
}
template <> struct FusedPub<double> {
  using T = FusedWord16;
  static __device__ __forceinline__ T word(double v, uint32_t tag) {
    return {(unsigned long long)__double_as_longlong(v), tag};
  }
  static __device__ __forceinline__ void gather(uint32_t c, uint32_t mine, uint32_t row, uint32_t n, uint32_t near,
                                                const T *far, double &v, T &w) {
    asm volatile(
        "{.reg .pred o, f; .reg .b128 t; setp.ge.u32 o, %3, %4; setp.lt.and.u32 f, %5, %6, o;"
        " mov.b128 t, {%1, %2}; @!o ld.shared.f64 %0, [%7]; @f ld.relaxed.gpu.global.b128 t, [%8];"
        " mov.b128 {%1, %2}, t;}"
        : "+d"(v), "+l"(w.lo), "+l"(w.hi)
        : "r"(c), "r"(mine), "r"(row), "r"(n), "r"(near), "l"(far)
        : "memory");
  }
  static __device__ __forceinline__ T get(const T *p) { return ld_word16(p); }
  static __device__ __forceinline__ void put(T *p, double v, uint32_t tag) { st_word16(p, word(v, tag).lo, tag); }
  static __device__ __forceinline__ uint32_t tag(T t) { return (uint32_t)t.hi; }
  static __device__ __forceinline__ double value(T t) { return __longlong_as_double((long long)t.lo); }
};

// A CTA's slices of the ns, `ctas` in all.
struct FusedSlices {
  int32_t first, count;
  __device__ FusedSlices(int64_t ns, int64_t cta, int64_t ctas)
      : first((int32_t)(ns * cta / ctas)), count((int32_t)(ns * (cta + 1) / ctas) - first) {}
};

// The matrix's distinct diagonals (column - row): d[0] and d[ND - 1] the lowest
// and the highest, the others between ascending and in [lo, hi].
struct FusedDiags {
  int32_t d[kFusedDiags], lo, hi;
};

// A row's values on the diagonals, kFusedDiags of them side by side.
template <typename V> struct FusedRow {
  static constexpr int kWords = kFusedDiags * (int)sizeof(V) / 16;
  uint4 w[kWords];
  __device__ __forceinline__ void load(const void *val, uint32_t row) {  // row * kWords < 2^32
#pragma unroll
    for (int k = 0; k < kWords; ++k) w[k] = __ldg(reinterpret_cast<const uint4 *>(val) + row * kWords + k);
  }
  template <int K>
  __device__ __forceinline__ typename std::conditional<sizeof(V) == 8, double, float>::type value() const {
    constexpr int kPer = 16 / (int)sizeof(V);
    const uint4 t = w[K / kPer];
    constexpr int e = K % kPer;
    if constexpr (sizeof(V) == 8) {
      return e ? __hiloint2double((int)t.w, (int)t.z) : __hiloint2double((int)t.y, (int)t.x);
    } else if constexpr (sizeof(V) == 4) {
      return __uint_as_float(e == 0 ? t.x : e == 1 ? t.y : e == 2 ? t.z : t.w);
    } else {
      const uint32_t u = e / 2 == 0 ? t.x : e / 2 == 1 ? t.y : e / 2 == 2 ? t.z : t.w;
      if constexpr (std::is_same<V, __half>::value) {
        const __half2 h = *reinterpret_cast<const __half2 *>(&u);
        return e & 1 ? __high2float(h) : __low2float(h);
      } else {
        return __uint_as_float(e & 1 ? u & 0xffff0000u : u << 16);
      }
    }
  }
};

// Distinct diagonals of the matrix into `set` (kFusedDiags values, kNoDiag when
// free); *overflow when there are more, or when a row's columns are not strictly
// ascending (a repeated column, unsorted rows): the copy by diagonals has one
// place per diagonal and takes a row's entries in order.
constexpr int32_t kNoDiag = INT32_MIN;
__global__ void fused_diags_kernel(int32_t n, const int32_t *__restrict__ rowPtr, const int32_t *__restrict__ colIdx,
                                   int32_t *set, int32_t *overflow) {
  __shared__ int32_t seen[kFusedDiags];
  if (threadIdx.x < kFusedDiags) seen[threadIdx.x] = kNoDiag;
  __syncthreads();
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
    if (*reinterpret_cast<volatile int32_t *>(overflow)) return;
    int32_t before = INT32_MIN;
    for (int32_t j = rowPtr[t]; j < rowPtr[t + 1]; ++j) {
      const int32_t c = colIdx[j], d = (int32_t)(c - t);
      if (c <= before) {
        *overflow = 1;
        return;
      }
      before = c;
      bool known = false;
#pragma unroll
      for (int k = 0; k < kFusedDiags; ++k) known |= *reinterpret_cast<volatile int32_t *>(seen + k) == d;
      if (known) continue;
      int at = 0;  // into the grid's set (looked at before it is written), then the CTA's
      for (; at < kFusedDiags; ++at) {
        int32_t old = *reinterpret_cast<volatile int32_t *>(set + at);
        if (old == kNoDiag) old = atomicCAS(set + at, kNoDiag, d);
        if (old == kNoDiag || old == d) break;
      }
      if (at == kFusedDiags) {
        *overflow = 1;
        return;
      }
      seen[at] = d;
    }
  }
}

// Fills the copy by diagonals: thread per slice row; a diagonal that the row
// lacks (and rows past n) gets 0.
template <typename V, bool SCALED>
__global__ void fused_fill_kernel(int32_t n, const int32_t *__restrict__ rowPtr, const int32_t *__restrict__ colIdx,
                                  const double *__restrict__ val, const int8_t *__restrict__ exps, FusedDiags D,
                                  V *__restrict__ out) {
  const int64_t rows = ((int64_t)n + 31) / 32 * 32;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < rows; t += (int64_t)gridDim.x * blockDim.x) {
    int32_t j = t < n ? rowPtr[t] : 0;
    const int32_t e = t < n ? rowPtr[t + 1] : 0;
#pragma unroll
    for (int k = 0; k < kFusedDiags; ++k) {
      double v = 0.0;
      if (j < e && colIdx[j] - t == D.d[k]) {
        v = val[j++];
        if (SCALED) v = ldexp(v, -(int)exps[t]);
      }
      if constexpr (sizeof(V) == 8)
        out[t * kFusedDiags + k] = v;
      else
        out[t * kFusedDiags + k] = from_float_lp<V>((float)v);
    }
  }
}

struct FusedGrid {
  CgSlot *slots;  // [2][kFusedMaxCtas]
  int32_t *err;
  unsigned long long epoch;
  double *part, *sum;  // shared: a partial per warp, a sum per polling warp
  int *dead;           // shared, 0 at the start
  uint32_t limit;      // LIMITED: polls of a grid sum
};

__device__ __forceinline__ bool fused_give_up(FusedGrid &G, uint32_t polls) {
  if ((polls & 1023u) != 0) return false;
  if (polls < kFusedPolls && *reinterpret_cast<volatile int32_t *>(G.err) == 0) return false;
  atomicExch(G.err, 1);
  *reinterpret_cast<volatile int *>(G.dead) = 1;
  return true;
}

// Sum over all threads of the grid (the same bits in every thread); the CTA's
// threads are in step on both sides.
template <int WARPS, bool LIMITED>
__device__ __forceinline__ double fused_sum(FusedGrid &G, double v) {
  constexpr int kPollWarps = kFusedMaxCtas / 32;
  static_assert(WARPS >= kPollWarps && WARPS <= 32, "a slot per thread, a partial per lane");
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  ++G.epoch;
  v = warp_sum(v);
  if (lane == 0) G.part[w] = v;
  __syncthreads();
  if (w < kPollWarps) {
    CgSlot *row = G.slots + (G.epoch & 1) * kFusedMaxCtas;
    if (w == 0) {
      const double t = warp_sum(lane < WARPS ? G.part[lane] : 0.0);
      if (lane == 0) st_word16(row + blockIdx.x, (unsigned long long)__double_as_longlong(t), G.epoch);
    }
    double got = 0.0;
    if (threadIdx.x < gridDim.x)
      for (uint32_t polls = 1;; ++polls) {
        const FusedWord16 t = ld_word16(row + threadIdx.x);
        got = __longlong_as_double((long long)t.lo);
        if (t.hi == G.epoch || fused_give_up(G, LIMITED && polls >= G.limit ? kFusedPolls : polls)) break;
      }
    got = warp_sum(got);
    if (lane == 0) G.sum[w] = got;
  }
  __syncthreads();
  double t = 0.0;
#pragma unroll
  for (int k = 0; k < kPollWarps; ++k) t += G.sum[k];
  return t;
}

// acc += sum of a row's values times p, in the diagonals' order.
template <int K, int ND, typename Row, typename VT>
__device__ __forceinline__ void fused_dot(const Row &a, const VT (&p)[ND], VT &acc) {
  if constexpr (K < ND) {
    acc = fma((VT)a.template value<K>(), p[K], acc);
    fused_dot<K + 1, ND>(a, p, acc);
  }
}

// ND: the diagonals looked at (the rest of the kFusedDiags are unused).
template <typename V, typename VT, int ND, int THREADS, bool LIMITED>
__global__ void __launch_bounds__(THREADS, 1)
    cg_fused_kernel(int32_t n, const void *__restrict__ val, FusedDiags D, const int8_t *__restrict__ exps,
                    VT *__restrict__ x, VT *__restrict__ r, VT *__restrict__ p_state, typename FusedPub<VT>::T *pub,
                    double *rr_part, int npart, double *sc, int iters, CgSlot *slots, unsigned long long *epoch_mem,
                    int32_t *err, uint32_t limit) {
  using Pub = FusedPub<VT>;
  using Vec = typename Vec16<VT>::T;
  constexpr int W = Vec16<VT>::W;
  constexpr bool kScaled = sizeof(V) == 2;
  constexpr int kWarps = THREADS / 32;
  extern __shared__ __align__(16) unsigned char fused_smem[];
  __shared__ double part[kWarps], sum[kFusedMaxCtas / 32];
  __shared__ int dead;
  const int lane = threadIdx.x & 31, w = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);  // uniform
  const int64_t ns = ((int64_t)n + 31) / 32;
  const FusedSlices T(ns, blockIdx.x, gridDim.x);
  const int32_t S = T.count, s_lo = T.first, row0 = s_lo * 32;
  const int32_t nloc = min(S * 32, n - row0);  // rows of the matrix; S * 32 with the padding
  const int32_t cap = (int32_t)((ns + gridDim.x - 1) / gridDim.x) * 32;
  VT *sx = reinterpret_cast<VT *>(fused_smem), *sr = sx + cap, *sp = sr + cap, *sq = sp + cap;
  const uint32_t sp_base = (uint32_t)__cvta_generic_to_shared(sp);
  typename Pub::T *pub0 = pub + row0;
  FusedGrid G{slots, err, *epoch_mem, part, sum, &dead, limit};
  if (threadIdx.x == 0) dead = 0;
  for (int32_t i = threadIdx.x; i < S * 32; i += THREADS) {  // padding rows stay 0
    const bool in = i < nloc;
    sx[i] = in ? x[row0 + i] : VT(0);
    sr[i] = in ? r[row0 + i] : VT(0);
    sp[i] = in ? p_state[row0 + i] : VT(0);
    sq[i] = VT(0);
  }
  double rr = 0.0;
  for (int i = threadIdx.x; i < npart; i += THREADS) rr += __ldcg(rr_part + i);
  rr = warp_sum(rr);
  if (lane == 0) part[w] = rr;
  __syncthreads();
  rr = warp_sum(lane < kWarps ? part[lane] : 0.0);
  double rr_prev = sc[1];
  __syncthreads();

  for (int it = 0; it < iters; ++it) {
    const double beta = (rr_prev != 0.0 && isfinite(rr)) ? rr / rr_prev : 0.0;
    const VT bt = (VT)beta;
    const uint32_t tag = (uint32_t)G.epoch + 1;
    FusedRow<V> e;
    int ex = 0;
    auto fetch = [&](int32_t sl) {
      e.load(val, row0 + sl * 32 + lane);
      if (kScaled) ex = exps[row0 + min(sl * 32 + lane, nloc - 1)];
    };
    if (w < S) fetch(w);  // in flight while p is formed
#pragma unroll 4
    for (int32_t i = threadIdx.x; i < S * 32; i += THREADS) {
      const VT pi = fma(bt, sp[i], sr[i]);
      sp[i] = pi;
      Pub::put(pub0 + i, pi, tag);
    }
    __syncthreads();
    double dot = 0.0;
    for (int32_t sl = w; sl < S; sl += kWarps) {
      const int32_t i = sl * 32 + lane;
      // p of the row's columns.  The inner diagonals of most slices lie among the
      // CTA's rows: shared memory; the outer ones (and all of them otherwise) are
      // told apart lane by lane.
      const uint32_t own = sp_base + (uint32_t)i * (uint32_t)sizeof(VT);
      VT near[ND];
      typename Pub::T g[ND];
      auto gather = [&](int k) {
        near[k] = VT(0);
        g[k] = Pub::word(VT(0), tag);
        Pub::gather((uint32_t)(i + D.d[k]), (uint32_t)(S * 32), (uint32_t)(row0 + i + D.d[k]), (uint32_t)n,
                    own + (uint32_t)D.d[k] * (uint32_t)sizeof(VT), pub0 + (i + D.d[k]), near[k], g[k]);
      };
      auto late = [&](int k) {
        for (uint32_t polls = 1; Pub::tag(g[k]) != tag && !fused_give_up(G, polls); ++polls)
          g[k] = Pub::get(pub0 + (i + D.d[k]));
      };
      auto take = [&](int k) {
        if ((uint32_t)(i + D.d[k]) >= (uint32_t)(S * 32)) near[k] = Pub::value(g[k]);
      };
      const bool inner = sl * 32 + D.lo >= 0 && sl * 32 + 32 + D.hi <= S * 32;  // warp-uniform
      gather(0);
      gather(ND - 1);
      if (inner) {
        const char *own_p = reinterpret_cast<const char *>(sp + i);
#pragma unroll
        for (int k = 1; k < ND - 1; ++k) near[k] = *reinterpret_cast<const VT *>(own_p + D.d[k] * (int)sizeof(VT));
      } else {
#pragma unroll
        for (int k = 1; k < ND - 1; ++k) gather(k);
      }
      const FusedRow<V> a = e;
      const float scale = kScaled ? pow2f(ex) : 1.f;
      if (sl + kWarps < S) fetch(sl + kWarps);  // in flight during this slice's gathers
      // one test for the usual case: everything has arrived
      if (Pub::tag(g[0]) != tag || Pub::tag(g[ND - 1]) != tag) {
        late(0);
        late(ND - 1);
      }
      take(0);
      take(ND - 1);
      if (!inner) {
#pragma unroll
        for (int k = 1; k < ND - 1; ++k) {
          late(k);
          take(k);
        }
      }
      VT acc = VT(0);
      fused_dot<0, ND>(a, near, acc);
      if constexpr (kScaled) acc *= scale;
      sq[i] = acc;  // 0 in a padding row
      dot += (double)acc * (double)sp[i];
    }
    const double pq = fused_sum<kWarps, LIMITED>(G, dot);
    if (dead) return;
    const double alpha = (pq != 0.0 && rr != 0.0 && isfinite(pq)) ? rr / pq : 0.0;
    const VT al = (VT)alpha;
    double s = 0.0;
    for (int32_t i = threadIdx.x * W; i < S * 32; i += THREADS * W) {
      const Vec p = *reinterpret_cast<const Vec *>(sp + i), q = *reinterpret_cast<const Vec *>(sq + i);
      Vec xv = *reinterpret_cast<Vec *>(sx + i), rv = *reinterpret_cast<Vec *>(sr + i);
#pragma unroll
      for (int k = 0; k < W; ++k) {
        vset(xv, k, fma(al, vget(p, k), vget(xv, k)));
        const VT ri = fma(-al, vget(q, k), vget(rv, k));
        vset(rv, k, ri);
        s += (double)ri * (double)ri;
      }
      *reinterpret_cast<Vec *>(sx + i) = xv;
      *reinterpret_cast<Vec *>(sr + i) = rv;
    }
    rr_prev = rr;
    rr = fused_sum<kWarps, LIMITED>(G, s);
    if (dead) return;
  }
  for (int32_t i = threadIdx.x; i < nloc; i += THREADS) {
    x[row0 + i] = sx[i];
    r[row0 + i] = sr[i];
    p_state[row0 + i] = sp[i];
  }
  if (blockIdx.x == 0) {
    for (int i = threadIdx.x; i < npart; i += THREADS) rr_part[i] = i == 0 ? rr : 0.0;
    if (threadIdx.x == 0) {
      sc[1] = rr_prev;
      sc[4] = rr;
      *epoch_mem = G.epoch;
    }
  }
}

// Kernel B: alpha = rr_k / p.q; x += alpha p; r -= alpha q; partials of r.r.
// 16-byte vector accesses (4 floats or 2 doubles per load), two in flight
// per thread; the scalar tail covers n not divisible by the vector width.
template <typename VT>
__global__ void __launch_bounds__(kCgThreads) cg_update_kernel(int32_t n, const double *__restrict__ pq_part,
                                                               int npart, const double *__restrict__ rr_slot,
                                                               VT *__restrict__ x, VT *__restrict__ r,
                                                               const VT *__restrict__ p, const VT *__restrict__ q,
                                                               double *__restrict__ rr_part) {
  using V = typename Vec16<VT>::T;
  constexpr int W = Vec16<VT>::W;
  constexpr int U = 2;
  __shared__ double smem[kCgThreads / 32];
  const int64_t nv = n / W;
  const int64_t stride = (int64_t)gridDim.x * kCgThreads;
  V *xv = reinterpret_cast<V *>(x);
  V *rv = reinterpret_cast<V *>(r);
  const V *pv = reinterpret_cast<const V *>(p);
  const V *qv = reinterpret_cast<const V *>(q);
  V P[U], Q[U], X[U], R[U];
  auto load = [&](int64_t i0) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i = i0 + u * stride;
      if (i < nv) {
        P[u] = pv[i];
        Q[u] = qv[i];
        X[u] = xv[i];
        R[u] = rv[i];
      }
    }
  };
  // the first pass's vectors do not depend on alpha: their loads are in
  // flight while the CTA sums the p.q partials
  const int64_t first = (int64_t)blockIdx.x * kCgThreads + threadIdx.x;
  load(first);
  const double pq = reduce_partials(pq_part, npart, smem);
  const double rr = *rr_slot;
  const double alpha = (pq != 0.0 && rr != 0.0 && isfinite(pq)) ? rr / pq : 0.0;
  const VT a = (VT)alpha;
  double s = 0.0;
  for (int64_t i0 = first; i0 < nv; i0 += U * stride) {
    if (i0 != first) load(i0);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i = i0 + u * stride;
      if (i < nv) {
#pragma unroll
        for (int k = 0; k < W; ++k) {
          vset(X[u], k, fma(a, vget(P[u], k), vget(X[u], k)));
          const VT ri = fma(-a, vget(Q[u], k), vget(R[u], k));
          vset(R[u], k, ri);
          s += (double)ri * (double)ri;
        }
        xv[i] = X[u];
        rv[i] = R[u];
      }
    }
  }
  for (int64_t i = nv * W + (int64_t)blockIdx.x * kCgThreads + threadIdx.x; i < n; i += stride) {
    x[i] = fma(a, p[i], x[i]);
    const VT ri = fma(-a, q[i], r[i]);
    r[i] = ri;
    s += (double)ri * (double)ri;
  }
  const double t = block_sum(s, smem);
  if (threadIdx.x == 0) rr_part[blockIdx.x] = t;
}

// ---------------------------------------------------------------------------
// Preconditioned CG (Jacobi: BS = 1; block-Jacobi: BS = 4 or 8 consecutive
// rows).  M^{-1} is stored in the iteration precision: dinv[n] for BS = 1,
// else the inverted diagonal blocks, BS*BS row-major per block (the last block
// padded with identity rows).  The preconditioned iteration keeps the two
// kernels: kernel A gathers z = M^{-1} r where it gathered r and reduces the
// r.z partials where it reduced r.r; the update kernel below also applies
// M^{-1} to the new residual and writes both the r.r partials (convergence
// checks) and the r.z partials (the next direction).
//
// One thread per group of G rows, G = 8 for 8x8 blocks and 4 otherwise (BS
// divides G, so blocks never straddle groups; 4 rows keep the FP64 kernel
// near 60 registers, 8 rows of five vectors needed 100 and halved the
// resident warps): 16-byte vector accesses for full groups, bounds-checked
// scalars for the last partial group.
template <int BS> struct PrecGroup { static constexpr int G = BS == 8 ? 8 : 4; };

template <typename VT, int G>
__device__ __forceinline__ void ldg_rows(const VT *__restrict__ p, VT (&v)[G]) {
  using V = typename Vec16<VT>::T;
  constexpr int W = Vec16<VT>::W;
  const V *pv = reinterpret_cast<const V *>(p);
#pragma unroll
  for (int u = 0; u < G / W; ++u) {
    const V t = pv[u];
#pragma unroll
    for (int k = 0; k < W; ++k) v[u * W + k] = vget(t, k);
  }
}

template <typename VT, int G>
__device__ __forceinline__ void stg_rows(VT *__restrict__ p, const VT (&v)[G]) {
  using V = typename Vec16<VT>::T;
  constexpr int W = Vec16<VT>::W;
  V *pv = reinterpret_cast<V *>(p);
#pragma unroll
  for (int u = 0; u < G / W; ++u) {
    V t;
#pragma unroll
    for (int k = 0; k < W; ++k) vset(t, k, v[u * W + k]);
    pv[u] = t;
  }
}

// z = M^{-1} r for the G-row group starting at row i0 (rows >= n hold r = 0).
template <typename VT, int BS, int G>
__device__ __forceinline__ void apply_minv(const VT *__restrict__ minv, int64_t i0, int32_t n, const VT (&r)[G],
                                           VT (&z)[G]) {
  if constexpr (BS == 1) {
    if (i0 + G <= n) {
      VT d[G];
      ldg_rows<VT, G>(minv + i0, d);
#pragma unroll
      for (int k = 0; k < G; ++k) z[k] = d[k] * r[k];
    } else {
#pragma unroll
      for (int k = 0; k < G; ++k) z[k] = i0 + k < n ? minv[i0 + k] * r[k] : VT(0);
    }
  } else {
    const int64_t nb = ((int64_t)n + BS - 1) / BS;
#pragma unroll
    for (int b = 0; b < G / BS; ++b) {
      const int64_t blk = i0 / BS + b;
      if (blk >= nb) {
#pragma unroll
        for (int i = 0; i < BS; ++i) z[b * BS + i] = VT(0);
        continue;
      }
      const VT *Mb = minv + blk * BS * BS;
#pragma unroll
      for (int i = 0; i < BS; ++i) {
        VT row[BS];
        ldg_rows<VT, BS>(Mb + i * BS, row);
        VT acc = VT(0);
#pragma unroll
        for (int j = 0; j < BS; ++j) acc = fma(row[j], r[b * BS + j], acc);
        z[b * BS + i] = acc;
      }
    }
  }
}

// UPDATE: alpha = rz / p.q; x += alpha p; r -= alpha q; then z = M^{-1} r,
// partials of r.r and r.z.  !UPDATE: z = M^{-1} r and r.z partials only
// (after the residual was replaced).
template <typename VT, int BS, bool UPDATE>
__global__ void __launch_bounds__(kCgThreads, 4) cg_update_prec_kernel(int32_t n, const double *__restrict__ pq_part,
                                                                    int npart, const double *__restrict__ rz_slot,
                                                                    VT *__restrict__ x, VT *__restrict__ r,
                                                                    VT *__restrict__ z, const VT *__restrict__ p,
                                                                    const VT *__restrict__ q,
                                                                    const VT *__restrict__ minv,
                                                                    double *__restrict__ rr_part,
                                                                    double *__restrict__ rz_part) {
  __shared__ double smem[kCgThreads / 32];
  VT a = VT(0);
  if constexpr (UPDATE) {
    const double pq = reduce_partials(pq_part, npart, smem);
    const double rz = *rz_slot;
    const double alpha = (pq != 0.0 && rz != 0.0 && isfinite(pq)) ? rz / pq : 0.0;
    a = (VT)alpha;
  }
  constexpr int G = PrecGroup<BS>::G;
  double srr = 0.0, srz = 0.0;
  const int64_t ng = ((int64_t)n + G - 1) / G;
  const int64_t stride = (int64_t)gridDim.x * kCgThreads;
  for (int64_t g = (int64_t)blockIdx.x * kCgThreads + threadIdx.x; g < ng; g += stride) {
    const int64_t i0 = g * G;
    const bool full = i0 + G <= n;
    VT R[G], Z[G];
    if (full) {
      ldg_rows<VT, G>(r + i0, R);
    } else {
#pragma unroll
      for (int k = 0; k < G; ++k) R[k] = i0 + k < n ? r[i0 + k] : VT(0);
    }
    if constexpr (UPDATE) {
      VT P[G], Q[G], X[G];
      if (full) {
        ldg_rows<VT, G>(p + i0, P);
        ldg_rows<VT, G>(q + i0, Q);
        ldg_rows<VT, G>(x + i0, X);
      } else {
#pragma unroll
        for (int k = 0; k < G; ++k) {
          const bool in = i0 + k < n;
          P[k] = in ? p[i0 + k] : VT(0);
          Q[k] = in ? q[i0 + k] : VT(0);
          X[k] = in ? x[i0 + k] : VT(0);
        }
      }
#pragma unroll
      for (int k = 0; k < G; ++k) {
        X[k] = fma(a, P[k], X[k]);
        R[k] = fma(-a, Q[k], R[k]);
        srr += (double)R[k] * (double)R[k];
      }
      if (full) {
        stg_rows<VT, G>(x + i0, X);
        stg_rows<VT, G>(r + i0, R);
      } else {
#pragma unroll
        for (int k = 0; k < G; ++k)
          if (i0 + k < n) {
            x[i0 + k] = X[k];
            r[i0 + k] = R[k];
          }
      }
    }
    apply_minv<VT, BS, G>(minv, i0, n, R, Z);
#pragma unroll
    for (int k = 0; k < G; ++k) srz += (double)R[k] * (double)Z[k];
    if (full) {
      stg_rows<VT, G>(z + i0, Z);
    } else {
#pragma unroll
      for (int k = 0; k < G; ++k)
        if (i0 + k < n) z[i0 + k] = Z[k];
    }
  }
  if constexpr (UPDATE) {
    const double t = block_sum(srr, smem);
    if (threadIdx.x == 0) rr_part[blockIdx.x] = t;
  }
  const double t2 = block_sum(srz, smem);
  if (threadIdx.x == 0) rz_part[blockIdx.x] = t2;
}

// M^{-1} from the CSR matrix: thread per block of BS rows; the block's
// entries (columns in the block's own range, found by binary search in the
// sorted row, duplicates summed) inverted by Gauss-Jordan elimination with
// partial pivoting in FP64.  A zero or non-finite pivot sets *bad.
template <typename VT, int BS>
__global__ void cg_minv_kernel(int32_t n, const int32_t *__restrict__ rowPtr, const int32_t *__restrict__ colIdx,
                               const double *__restrict__ val, VT *__restrict__ minv, int32_t *__restrict__ bad) {
  const int64_t nb = ((int64_t)n + BS - 1) / BS;
  for (int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += (int64_t)gridDim.x * blockDim.x) {
    double M[BS][BS], I[BS][BS];
    const int64_t lo = b * BS;
    for (int i = 0; i < BS; ++i)
      for (int j = 0; j < BS; ++j) {
        M[i][j] = 0.0;
        I[i][j] = i == j ? 1.0 : 0.0;
      }
    for (int i = 0; i < BS; ++i) {
      const int64_t row = lo + i;
      if (row >= n) {
        M[i][i] = 1.0;  // padding of the last block
        continue;
      }
      int32_t s = rowPtr[row], e = rowPtr[row + 1];
      while (s < e) {  // first column >= lo
        const int32_t m = s + ((e - s) >> 1);
        if (colIdx[m] < lo)
          s = m + 1;
        else
          e = m;
      }
      for (int32_t j = s; j < rowPtr[row + 1] && colIdx[j] < lo + BS; ++j) M[i][colIdx[j] - lo] += val[j];
    }
    bool ok = true;
    for (int c = 0; c < BS && ok; ++c) {
      int piv = c;
      for (int i = c + 1; i < BS; ++i)
        if (fabs(M[i][c]) > fabs(M[piv][c])) piv = i;
      if (!(fabs(M[piv][c]) > 0.0) || !isfinite(M[piv][c])) {
        ok = false;
        break;
      }
      if (piv != c)
        for (int j = 0; j < BS; ++j) {
          double t = M[c][j];
          M[c][j] = M[piv][j];
          M[piv][j] = t;
          t = I[c][j];
          I[c][j] = I[piv][j];
          I[piv][j] = t;
        }
      const double inv = 1.0 / M[c][c];
      for (int j = 0; j < BS; ++j) {
        M[c][j] *= inv;
        I[c][j] *= inv;
      }
      for (int i = 0; i < BS; ++i)
        if (i != c) {
          const double f = M[i][c];
          if (f != 0.0)
            for (int j = 0; j < BS; ++j) {
              M[i][j] -= f * M[c][j];
              I[i][j] -= f * I[c][j];
            }
        }
    }
    if (!ok) atomicExch(bad, 1);
    for (int i = 0; i < BS; ++i)
      for (int j = 0; j < BS; ++j) minv[b * BS * BS + i * BS + j] = (VT)(ok ? I[i][j] : (i == j ? 1.0 : 0.0));
  }
}

// FP64 true residual r = b - A x, a row per thread and the grid over all rows:
// the row's entries, then their x gathers, each loaded together.  (With the
// norms below in the same kernel and one wave of CTAs, each thread's rows were a
// serial chain of cold loads: Poisson 128^3 150 us, now 49 and 11.)
__global__ void __launch_bounds__(kCgThreads) cg_residual_kernel(int32_t n, const int32_t *__restrict__ rowPtr,
                                                                 const int32_t *__restrict__ colIdx,
                                                                 const double *__restrict__ val,
                                                                 const double *__restrict__ b,
                                                                 const double *__restrict__ x,
                                                                 double *__restrict__ r) {
  const int64_t i = (int64_t)blockIdx.x * kCgThreads + threadIdx.x;
  if (i >= n) return;
  const int32_t s = rowPtr[i], e = rowPtr[i + 1];
  int32_t c[kRowFirst];
  double a[kRowFirst], xv[kRowFirst];
#pragma unroll
  for (int k = 0; k < kRowFirst; ++k) {
    c[k] = s + k < e ? colIdx[s + k] : -1;
    a[k] = s + k < e ? val[s + k] : 0.0;
  }
#pragma unroll
  for (int k = 0; k < kRowFirst; ++k) xv[k] = c[k] >= 0 ? __ldg(x + c[k]) : 0.0;
  double acc = 0.0;
#pragma unroll
  for (int k = 0; k < kRowFirst; ++k)
    if (c[k] >= 0) acc = fma(a[k], xv[k], acc);
  for (int32_t j = s + kRowFirst; j < e; ++j) acc = fma(val[j], __ldg(x + colIdx[j]), acc);
  r[i] = b[i] - acc;
}

// Partials of ||r||^2; optionally also the inner-precision copy r_lp = (VT) r
// and its partials (reliable update), and the partials of ||r - r_lp_old||^2,
// the distance of the true residual from the iterated one it replaces
// (part_dev, may be null).
template <typename VT>
__global__ void __launch_bounds__(kCgThreads) cg_norm_kernel(int32_t n, const double *__restrict__ r,
                                                             VT *__restrict__ r_lp, double *__restrict__ part,
                                                             double *__restrict__ part_lp,
                                                             double *__restrict__ part_dev = nullptr) {
  __shared__ double smem[kCgThreads / 32];
  double nrm = 0.0, nrm_lp = 0.0, dev = 0.0;
  const int64_t stride = (int64_t)gridDim.x * kCgThreads;
#pragma unroll 4
  for (int64_t i = (int64_t)blockIdx.x * kCgThreads + threadIdx.x; i < n; i += stride) {
    const double ri = r[i];
    nrm += ri * ri;
    if (r_lp) {
      if (part_dev) {
        const double d = ri - (double)r_lp[i];
        dev += d * d;
      }
      const VT v = (VT)ri;
      r_lp[i] = v;
      nrm_lp += (double)v * (double)v;
    }
  }
  double t = block_sum(nrm, smem);
  if (threadIdx.x == 0) part[blockIdx.x] = t;
  if (r_lp) {
    t = block_sum(nrm_lp, smem);
    if (threadIdx.x == 0) part_lp[blockIdx.x] = t;
  }
  if (part_dev) {
    t = block_sum(dev, smem);
    if (threadIdx.x == 0) part_dev[blockIdx.x] = t;
  }
}

// x64 += x_lp; x_lp = 0 (reliable update of the solution).
template <typename VT>
__global__ void cg_fold_kernel(int32_t n, VT *__restrict__ x_lp, double *__restrict__ x) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    x[i] += (double)x_lp[i];
    x_lp[i] = VT(0);
  }
}

// ---------------------------------------------------------------------------
// Flexible outer iteration for the mixed modes (FCG(1), one previous
// direction): the inner low-precision (P)CG, run until its residual has
// dropped by reliable_delta, is the preconditioner z = B(r) of an FP64 CG on
// the FP64 matrix.  Because B changes from step to step (and the inner matrix
// is only an approximation of A), the new direction is A-orthogonalised
// against the previous one explicitly: p = z - (z.q_prev / p_prev.q_prev) p_prev,
// q = A p, alpha = p.r / p.q.  Unlike residual replacement, the outer Krylov
// step keeps converging when the low-precision matrix is far from A.
//
// F1: z = (double) x_lp; x_lp = 0; partials of z.q_prev.
__global__ void __launch_bounds__(kCgThreads) fcg_z_kernel(int32_t n, float *__restrict__ x_lp,
                                                           double *__restrict__ z, const double *__restrict__ q_prev,
                                                           double *__restrict__ part) {
  __shared__ double smem[kCgThreads / 32];
  double s = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * kCgThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kCgThreads) {
    const double zi = (double)x_lp[i];
    x_lp[i] = 0.f;
    z[i] = zi;
    s += zi * q_prev[i];
  }
  const double t = block_sum(s, smem);
  if (threadIdx.x == 0) part[blockIdx.x] = t;
}

// F2: p = z - gamma p_prev, gamma = z.q_prev / pq_prev (0 on the first step).
__global__ void __launch_bounds__(kCgThreads) fcg_dir_kernel(int32_t n, const double *__restrict__ part, int npart,
                                                             const double *__restrict__ pq_prev_slot,
                                                             const double *__restrict__ z, double *__restrict__ p) {
  __shared__ double smem[kCgThreads / 32];
  const double zq = reduce_partials(part, npart, smem);
  const double pq_prev = *pq_prev_slot;
  const double gamma = (pq_prev != 0.0 && isfinite(zq)) ? zq / pq_prev : 0.0;
  for (int64_t i = (int64_t)blockIdx.x * kCgThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kCgThreads)
    p[i] = gamma != 0.0 ? fma(-gamma, p[i], z[i]) : z[i];
}

// F3: q = A p (FP64 CSR); partials of p.q and p.r.
__global__ void __launch_bounds__(kCgThreads) fcg_spmv_kernel(int32_t n, const int32_t *__restrict__ rowPtr,
                                                              const int32_t *__restrict__ colIdx,
                                                              const double *__restrict__ val,
                                                              const double *__restrict__ p, double *__restrict__ q,
                                                              const double *__restrict__ r,
                                                              double *__restrict__ part_pq,
                                                              double *__restrict__ part_pr) {
  __shared__ double smem[kCgThreads / 32];
  double spq = 0.0, spr = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * kCgThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kCgThreads) {
    const int32_t s0 = rowPtr[i], e0 = rowPtr[i + 1];
    int32_t c[kRowFirst];
    double a[kRowFirst];
#pragma unroll
    for (int k = 0; k < kRowFirst; ++k) {
      c[k] = s0 + k < e0 ? colIdx[s0 + k] : -1;
      a[k] = s0 + k < e0 ? val[s0 + k] : 0.0;
    }
    double acc = 0.0;
#pragma unroll
    for (int k = 0; k < kRowFirst; ++k)
      if (c[k] >= 0) acc = fma(a[k], __ldg(p + c[k]), acc);
    for (int32_t j = s0 + kRowFirst; j < e0; ++j) acc = fma(val[j], __ldg(p + colIdx[j]), acc);
    q[i] = acc;
    spq += p[i] * acc;
    spr += p[i] * r[i];
  }
  double t = block_sum(spq, smem);
  if (threadIdx.x == 0) part_pq[blockIdx.x] = t;
  t = block_sum(spr, smem);
  if (threadIdx.x == 0) part_pr[blockIdx.x] = t;
}

// F4: alpha = p.r / p.q; x += alpha p; r -= alpha q; r_lp = (float) r;
// partials of r.r and r_lp.r_lp; p.q kept in *pq_slot for the next F2.
__global__ void __launch_bounds__(kCgThreads) fcg_update_kernel(int32_t n, const double *__restrict__ part_pq,
                                                                const double *__restrict__ part_pr, int npart,
                                                                double *__restrict__ pq_slot,
                                                                double *__restrict__ x, double *__restrict__ r,
                                                                const double *__restrict__ p,
                                                                const double *__restrict__ q,
                                                                float *__restrict__ r_lp,
                                                                double *__restrict__ part_rr,
                                                                double *__restrict__ part_rr_lp) {
  __shared__ double smem[kCgThreads / 32];
  const double pq = reduce_partials(part_pq, npart, smem);
  const double pr = reduce_partials(part_pr, npart, smem);
  const double alpha = (pq > 0.0 && isfinite(pq) && isfinite(pr)) ? pr / pq : 0.0;
  double s = 0.0, sl = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * kCgThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kCgThreads) {
    x[i] = fma(alpha, p[i], x[i]);
    const double ri = fma(-alpha, q[i], r[i]);
    r[i] = ri;
    const float rl = (float)ri;
    r_lp[i] = rl;
    s += ri * ri;
    sl += (double)rl * (double)rl;
  }
  double t = block_sum(s, smem);
  if (threadIdx.x == 0) part_rr[blockIdx.x] = t;
  t = block_sum(sl, smem);
  if (threadIdx.x == 0) {
    part_rr_lp[blockIdx.x] = t;
    if (blockIdx.x == 0) *pq_slot = (pq > 0.0 && isfinite(pq)) ? pq : 0.0;
  }
}

__global__ void sum_partials_kernel(const double *__restrict__ part, int npart, double *__restrict__ out) {
  __shared__ double smem[kCgThreads / 32];
  const double s = reduce_partials(part, npart, smem);
  if (threadIdx.x == 0) *out = s;
}

// ---------------------------------------------------------------------------
// Low-precision SELL-32 copy of the matrix.
__global__ void sell_len_kernel(int32_t n, const int32_t *__restrict__ rowPtr, int32_t *__restrict__ slice_len) {
  const int64_t ns = ((int64_t)n + 31) / 32;
  for (int64_t sl = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; sl < ns; sl += (int64_t)gridDim.x * blockDim.x) {
    int32_t m = 0;
    for (int64_t r = sl * 32; r < n && r < sl * 32 + 32; ++r) m = max(m, rowPtr[r + 1] - rowPtr[r]);
    slice_len[sl] = m;
  }
}

// One power-of-two exponent per row: the row's largest magnitude scaled into [1, 2).
__global__ void row_exp_kernel(int32_t n, const int32_t *__restrict__ rowPtr, const double *__restrict__ val,
                               int8_t *__restrict__ exps) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
    double m = 0.0;
    for (int32_t j = rowPtr[r]; j < rowPtr[r + 1]; ++j) m = fmax(m, fabs(val[j]));
    int e = 0;
    if (m > 0.0) {
      frexp(m, &e);  // m = f * 2^e, f in [0.5, 1)
      e -= 1;
    }
    exps[r] = (int8_t)(e < -100 ? -100 : (e > 100 ? 100 : e));
  }
}

// Thread per (slice row): its entries (scaled, converted) and columns (int16
// offsets or int32) into the slice; padding = value 0, column = the row
// itself (rows past n in the last slice: column 0, never gathered).
template <typename V, bool SCALED, bool D16, bool PACKED>
__global__ void sell_fill_kernel(int32_t n, const int32_t *__restrict__ rowPtr, const int32_t *__restrict__ colIdx,
                                 const double *__restrict__ val, const int32_t *__restrict__ slice_len,
                                 const int64_t *__restrict__ slice_off, const int8_t *__restrict__ exps,
                                 V *__restrict__ out, void *__restrict__ cols) {
  const int64_t ns = ((int64_t)n + 31) / 32;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < ns * 32; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t sl = t >> 5, lane = t & 31;
    const int64_t self = t < n ? t : 0;
    const int32_t s0 = t < n ? rowPtr[t] : 0, e0 = t < n ? rowPtr[t + 1] : 0;
    for (int32_t k = 0; k < slice_len[sl]; ++k) {
      const int64_t j = slice_off[sl] + (int64_t)k * 32 + lane;
      double v = 0.0;
      int64_t c = self;
      if (s0 + k < e0) {
        v = val[s0 + k];
        c = colIdx[s0 + k];
        if (SCALED) v = ldexp(v, -(int)exps[t]);
      }
      V lv;
      if constexpr (sizeof(V) == 8)
        lv = v;  // the FP64 copy keeps the values exactly
      else
        lv = from_float_lp<V>((float)v);
      const int64_t d = c - self;
      if (PACKED) {
        unsigned short vb;
        memcpy(&vb, &lv, sizeof(vb));
        reinterpret_cast<uint32_t *>(out)[j] = (uint32_t)vb | ((uint32_t)(uint16_t)(int16_t)d << 16);
      } else {
        out[j] = lv;
        if (D16)
          reinterpret_cast<int16_t *>(cols)[j] = (int16_t)d;
        else
          reinterpret_cast<int32_t *>(cols)[j] = (int32_t)c;
      }
    }
  }
}

__global__ void cg_delta_check_kernel(int32_t n, const int32_t *__restrict__ rowPtr,
                                      const int32_t *__restrict__ colIdx, int32_t *__restrict__ bad) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    for (int32_t j = rowPtr[i]; j < rowPtr[i + 1]; ++j) {
      const int64_t d = (int64_t)colIdx[j] - i;
      if (d < -32768 || d > 32767) {
        atomicExch(bad, 1);
        break;
      }
    }
}

__global__ void f64_to_f32_kernel(int64_t n, const double *__restrict__ a, float *__restrict__ b) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    b[i] = (float)a[i];
}


}  // namespace bsp

// ---------------------------------------------------------------------------
struct bsp_cg_plan_s {
  int32_t n = 0, nnz = 0;
  bsp_cg_options opt{};
  const int32_t *rowPtr = nullptr, *colIdx = nullptr;
  const double *val = nullptr;
  // low-precision copy of the matrix (mixed modes)
  void *lp_val = nullptr;
  int8_t *exps = nullptr;
  void *lp_cols = nullptr;     // int16 offsets or int32 columns (unpacked SELL)
  int32_t *slice_len = nullptr;
  int64_t *slice_off = nullptr;
  int32_t sell_uniform = 0;    // > 0: all slices padded to this length
  bool delta16 = false;
  bool sell64 = false;         // FP64 mode iterates on an FP64 SELL-32 copy
  // FP64 state
  double *x64 = nullptr, *r64 = nullptr;
  // iteration vectors: FP64 (mode FP64) or FP32 (mixed); p ping-pongs
  void *x = nullptr, *r = nullptr, *p[2] = {nullptr, nullptr}, *q = nullptr;
  double *part_pq = nullptr, *part_rr = nullptr, *part_res = nullptr;
  // preconditioning: prec_bs = 0 (none), 1 (Jacobi), 4 or 8 (block-Jacobi)
  int prec_bs = 0;
  int lpr = 1;  // FP64 mode: lanes per row of the direction/SpMV kernel
  void *z = nullptr, *minv = nullptr;
  double *part_rz = nullptr;
  // flexible outer iteration (mixed modes): FP64 p, q, z; r64 holds the
  // FP64 residual; partials of z.q_prev and p.r
  double *p64 = nullptr, *q64 = nullptr, *z64 = nullptr;
  double *part_zq = nullptr, *part_pr = nullptr;
  int64_t bytes_outer = 0;
  double *sc = nullptr, *h_sc = nullptr;  // [0],[1] rr slots, [2] ||b-Ax||^2, [3] ||b||^2, [4] rr after a chunk,
                                          // [8] error flag, [9] epoch of the fused iteration
  int grid = 0;    // update, residual and reduction kernels (writers of the rr partials)
  int grid_a = 0;  // direction/SpMV kernel (writer of the p.q partials)
  // fused iteration (one cooperative launch per chunk): 0 CTAs = not used
  int fused_ctas = 0;
  size_t fused_smem = 0;
  bsp::CgSlot *slots = nullptr;
  void *pub = nullptr;  // published p with tags
  void *fused_val = nullptr;  // the matrix by diagonals
  bsp::FusedDiags fused_diags{};
  int fused_nd = 0;
  uint32_t fused_polls = bsp::kFusedPolls;
  cudaGraphExec_t graph = nullptr;
  cudaStream_t graph_stream = nullptr;
  int64_t bytes_iter = 0, bytes_chunk = 0, bytes_residual = 0;
};

namespace bsp {

constexpr int kCgMaxCtasPerSm = 2048 / kCgThreads;
constexpr int kCgScalars = 10;
// 64 registers a thread in FP32; an FP64 thread holds twice the bytes in flight
constexpr int kFusedThreads32 = 1024, kFusedThreads64 = 512;
// Mixed modes: a replaced (true) residual whose distance from the iterated
// one exceeds kCgDeviation x its norm, or an iterated residual above kCgGrowth
// x the last true one, marks the low-precision matrix as too far from A for
// residual replacement (AUTO then switches to the flexible outer iteration).
// Measured: <= 0.006 where replacement keeps the FP64 iteration count, >= 0.13
// where it costs 1.5x-30x more iterations.
constexpr double kCgDeviation = 0.1;
constexpr double kCgGrowth = 1e4;
// Mixed modes: this many residual replacements in a row without a new lowest
// true residual end the solve (BSP_ERR_NOT_CONVERGED).
constexpr int kCgNoProgress = 6;
// Mixed modes: this many chunks without the inner drop force a residual
// replacement / outer step (an inner iteration that stagnates).
constexpr int kCgInnerChunks = 32;

// Resident CTAs per SM of the direction/SpMV kernel (a) and of the update
// kernel (b).
template <typename V, typename VT, bool SC, bool D16>
static void cg_occupancy(int &a, int &b) {
  a = b = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, cg_dir_spmv_kernel<V, VT, SC, D16>, kCgThreads, 0) !=
      cudaSuccess)
    a = 4;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, cg_update_kernel<VT>, kCgThreads, 0) != cudaSuccess) b = 4;
  a = a < 1 ? 1 : (a > kCgMaxCtasPerSm ? kCgMaxCtasPerSm : a);
  b = b < 1 ? 1 : (b > kCgMaxCtasPerSm ? kCgMaxCtasPerSm : b);
}

// One resident wave (grid-stride loops inside).
static int cg_grid(int32_t n, int occ) {
  int64_t g = ceil_div(n, kCgThreads);
  const int64_t cap = (int64_t)sm_count() * occ;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return (int)g;
}

static bool cg_mixed(const bsp_cg_plan_s *P) { return P->opt.mode != BSP_CG_FP64; }

static void cg_plan_occupancy(const bsp_cg_plan_s *P, int &a, int &b) {
  const bool d = P->delta16;
  switch (P->opt.mode) {
    case BSP_CG_FP64:
      return P->sell64 ? cg_occupancy<double, double, false, true>(a, b)
                       : cg_occupancy<double, double, false, false>(a, b);
    case BSP_CG_MIXED_F32:
      return d ? cg_occupancy<float, float, false, true>(a, b) : cg_occupancy<float, float, false, false>(a, b);
    case BSP_CG_MIXED_F16:
      return d ? cg_occupancy<__half, float, true, true>(a, b) : cg_occupancy<__half, float, true, false>(a, b);
    default:
      return d ? cg_occupancy<__nv_bfloat16, float, true, true>(a, b)
               : cg_occupancy<__nv_bfloat16, float, true, false>(a, b);
  }
}

template <typename V, typename VT, bool SC, bool D16, int LPR = 1>
static void launch_iter(bsp_cg_plan_s *P, int k, cudaStream_t s) {
  constexpr bool csr = sizeof(V) == 8 && !D16;  // FP64 CSR; the other forms read the SELL copy
  CgMat<V, VT, SC, D16> A{P->rowPtr, csr ? (const void *)P->colIdx : (const void *)P->lp_cols,
                           (const V *)(csr ? (const void *)P->val : P->lp_val), P->exps,
                           P->slice_len, P->slice_off, P->sell_uniform};
  VT *r = (VT *)P->r, *x = (VT *)P->x, *q = (VT *)P->q;
  VT *pp = (VT *)P->p[k & 1], *pn = (VT *)P->p[(k + 1) & 1];
  const int g = P->grid, ga = P->grid_a;
  if (P->prec_bs == 0) {
    cg_dir_spmv_kernel<V, VT, SC, D16, LPR><<<ga, kCgThreads, 0, s>>>(P->n, A, r, pp, pn, q, P->part_rr, g,
                                                                  P->sc + ((k + 1) & 1), P->sc + (k & 1),
                                                                  P->part_pq);
    cg_update_kernel<VT><<<g, kCgThreads, 0, s>>>(P->n, P->part_pq, ga, P->sc + (k & 1), x, r, pn, q, P->part_rr);
    return;
  }
  // preconditioned: directions from z, r.z in the scalar slots
  VT *z = (VT *)P->z;
  const VT *mi = (const VT *)P->minv;
  cg_dir_spmv_kernel<V, VT, SC, D16, LPR><<<ga, kCgThreads, 0, s>>>(P->n, A, z, pp, pn, q, P->part_rz, g,
                                                                P->sc + ((k + 1) & 1), P->sc + (k & 1),
                                                                P->part_pq);
  const double *sl = P->sc + (k & 1);
  switch (P->prec_bs) {
    case 1:
      cg_update_prec_kernel<VT, 1, true><<<g, kCgThreads, 0, s>>>(P->n, P->part_pq, ga, sl, x, r, z, pn, q, mi,
                                                                   P->part_rr, P->part_rz);
      break;
    case 4:
      cg_update_prec_kernel<VT, 4, true><<<g, kCgThreads, 0, s>>>(P->n, P->part_pq, ga, sl, x, r, z, pn, q, mi,
                                                                   P->part_rr, P->part_rz);
      break;
    default:
      cg_update_prec_kernel<VT, 8, true><<<g, kCgThreads, 0, s>>>(P->n, P->part_pq, ga, sl, x, r, z, pn, q, mi,
                                                                   P->part_rr, P->part_rz);
  }
}

// z = M^{-1} r and the r.z partials, after the residual was replaced.
template <typename VT>
static void launch_prec(bsp_cg_plan_s *P, cudaStream_t s) {
  VT *r = (VT *)P->r, *z = (VT *)P->z;
  const VT *mi = (const VT *)P->minv;
  const int g = P->grid;
  switch (P->prec_bs) {
    case 1:
      cg_update_prec_kernel<VT, 1, false><<<g, kCgThreads, 0, s>>>(P->n, nullptr, 0, nullptr, nullptr, r, z, nullptr,
                                                                    nullptr, mi, nullptr, P->part_rz);
      break;
    case 4:
      cg_update_prec_kernel<VT, 4, false><<<g, kCgThreads, 0, s>>>(P->n, nullptr, 0, nullptr, nullptr, r, z, nullptr,
                                                                    nullptr, mi, nullptr, P->part_rz);
      break;
    default:
      cg_update_prec_kernel<VT, 8, false><<<g, kCgThreads, 0, s>>>(P->n, nullptr, 0, nullptr, nullptr, r, z, nullptr,
                                                                    nullptr, mi, nullptr, P->part_rz);
  }
}

static bsp_status cg_iteration(bsp_cg_plan_s *P, int k, cudaStream_t s) {
  if (P->sell64) {
    launch_iter<double, double, false, true>(P, k, s);
  } else if (!cg_mixed(P)) {
    switch (P->lpr) {
      case 2: launch_iter<double, double, false, false, 2>(P, k, s); break;
      case 4: launch_iter<double, double, false, false, 4>(P, k, s); break;
      case 8: launch_iter<double, double, false, false, 8>(P, k, s); break;
      default: launch_iter<double, double, false, false, 1>(P, k, s);
    }
  } else {
    const bool d = P->delta16;
    switch (P->opt.mode) {
      case BSP_CG_MIXED_F32:
        d ? launch_iter<float, float, false, true>(P, k, s) : launch_iter<float, float, false, false>(P, k, s);
        break;
      case BSP_CG_MIXED_F16:
        d ? launch_iter<__half, float, true, true>(P, k, s) : launch_iter<__half, float, true, false>(P, k, s);
        break;
      default:
        d ? launch_iter<__nv_bfloat16, float, true, true>(P, k, s)
          : launch_iter<__nv_bfloat16, float, true, false>(P, k, s);
    }
  }
  BSP_LAUNCH_CHECK();
  return BSP_OK;
}

// `check_every` iterations (even) followed by rr -> sc[4].
static bsp_status cg_chunk(bsp_cg_plan_s *P, cudaStream_t s) {
  for (int k = 0; k < P->opt.check_every; ++k) BSP_TRY(cg_iteration(P, k, s));
  sum_partials_kernel<<<1, kCgThreads, 0, s>>>(P->part_rr, P->grid, P->sc + 4);
  BSP_LAUNCH_CHECK();
  return BSP_OK;
}

static size_t fused_pub_bytes(const bsp_cg_plan_s *P);

// The two-kernel iteration's copy of the matrix: SELL-32 in the mixed modes and, where
// its rows are short and uniform, in FP64 (else FP64 stays on the CSR arrays).
#define BSP_CG_ALLOC(x)                                                                   \
  do {                                                                                    \
    cudaError_t e_ = (x);                                                                 \
    if (e_ != cudaSuccess) {                                                              \
      set_error(std::string("bsp_cg_create: ") + #x + " -> " + cudaGetErrorString(e_));   \
      return BSP_ERR_ALLOC;                                                               \
    }                                                                                     \
  } while (0)
static bsp_status two_kernel_setup(bsp_cg_plan_s *P, cudaStream_t s, int64_t *mat_bytes) {
  const int32_t n = P->n;
  const int32_t *rowPtr = P->rowPtr, *colIdx = P->colIdx;
  const bool mixed = cg_mixed(P);
  if (!mixed && P->lpr != 1) return BSP_OK;
  int64_t padded = 0;
  // SELL-32 slices: lengths on the device, offsets summed on the host
  const int64_t ns = ceil_div(n, 32);
  BSP_TRY(dalloc(&P->slice_len, (size_t)ns, s));
  BSP_TRY(dalloc(&P->slice_off, (size_t)ns + 1, s));
  const unsigned gs = (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(ns, 256), (int64_t)sm_count() * 16));
  sell_len_kernel<<<gs, 256, 0, s>>>(n, rowPtr, P->slice_len);
  std::vector<int32_t> hlen((size_t)ns);
  std::vector<int64_t> hoff((size_t)ns + 1, 0);
  BSP_CG_ALLOC(cudaMemcpyAsync(hlen.data(), P->slice_len, sizeof(int32_t) * ns, cudaMemcpyDeviceToHost, s));
  BSP_CG_ALLOC(cudaStreamSynchronize(s));
  // When padding every slice to the longest costs at most 1/32 more
  // storage (stencils, banded matrices), the direction kernel computes a
  // slice's offset instead of loading its length and offset.
  int32_t lmax = 0;
  int64_t natural = 0;
  for (int64_t k = 0; k < ns; ++k) {
    lmax = std::max(lmax, hlen[k]);
    natural += 32 * (int64_t)hlen[k];
  }
  if (lmax > 0 && ns * 32 * (int64_t)lmax <= natural + natural / 32) {
    std::fill(hlen.begin(), hlen.end(), lmax);
    BSP_CG_ALLOC(cudaMemcpyAsync(P->slice_len, hlen.data(), sizeof(int32_t) * ns, cudaMemcpyHostToDevice, s));
    P->sell_uniform = lmax;
  }
  for (int64_t k = 0; k < ns; ++k) hoff[k + 1] = hoff[k] + 32 * (int64_t)hlen[k];
  padded = hoff[ns];
  if (padded >= ((int64_t)1 << 31)) {
    if (mixed) {
      set_error("bsp_cg_create: the padded low-precision matrix needs >= 2^31 entries");
      return BSP_ERR_UNSUPPORTED;
    }
    P->sell_uniform = 0;  // FP64 stays on the CSR arrays
  }
  BSP_CG_ALLOC(cudaMemcpyAsync(P->slice_off, hoff.data(), sizeof(int64_t) * (ns + 1), cudaMemcpyHostToDevice, s));
  int32_t *bad = nullptr;
  BSP_TRY(dalloc(&bad, 1, s));
  cudaMemsetAsync(bad, 0, sizeof(int32_t), s);
  int64_t gr = ceil_div(n, 256);
  if (gr > (int64_t)sm_count() * 32) gr = (int64_t)sm_count() * 32;
  cg_delta_check_kernel<<<(unsigned)gr, 256, 0, s>>>(n, rowPtr, colIdx, bad);
  int32_t h_bad = 1;
  BSP_TRY(read_i32(bad, &h_bad, s));
  dfree(bad, s);
  P->delta16 = !h_bad;
  P->sell64 = !mixed && P->delta16 && P->sell_uniform > 0;
  if (!mixed && !P->sell64) {  // FP64 stays on the CSR arrays
    dfree(P->slice_len, s);
    dfree(P->slice_off, s);
    P->slice_len = nullptr;
    P->slice_off = nullptr;
    P->sell_uniform = 0;
  }
  if (!mixed && !P->sell64) return BSP_OK;
  {
    const bool scaled = mixed && P->opt.mode != BSP_CG_MIXED_F32;
    const size_t vsz = !mixed ? 8 : P->opt.mode == BSP_CG_MIXED_F32 ? 4 : 2;
    const bool packed = scaled && P->delta16;
    if (P->sell64) {
      // the FP64 copy is an optimisation: without room for it, stay on CSR
      const size_t ne = (size_t)(padded > 0 ? padded : 1);
      if (pool_malloc(reinterpret_cast<void **>(&P->lp_val), 8 * ne, s) != cudaSuccess ||
          pool_malloc(reinterpret_cast<void **>(&P->lp_cols), 2 * ne, s) != cudaSuccess) {
        cudaGetLastError();
        if (P->lp_val) pool_free(P->lp_val, s);
        if (P->lp_cols) pool_free(P->lp_cols, s);
        P->lp_val = P->lp_cols = nullptr;
        dfree(P->slice_len, s);
        dfree(P->slice_off, s);
        P->slice_len = nullptr;
        P->slice_off = nullptr;
        P->sell_uniform = 0;
        P->sell64 = false;
      }
    } else {
      BSP_CG_ALLOC(pool_malloc(reinterpret_cast<void **>(&P->lp_val), (packed ? 4 : vsz) * (size_t)(padded > 0 ? padded : 1), s));
      if (!packed)
        BSP_CG_ALLOC(pool_malloc(reinterpret_cast<void **>(&P->lp_cols), (P->delta16 ? 2 : 4) * (size_t)(padded > 0 ? padded : 1), s));
    }
  }
  if (mixed || P->sell64) {
    const bool scaled = mixed && P->opt.mode != BSP_CG_MIXED_F32;
    const size_t vsz = !mixed ? 8 : P->opt.mode == BSP_CG_MIXED_F32 ? 4 : 2;
    const int64_t ns = ceil_div(n, 32);
    const bool packed = scaled && P->delta16;
    int64_t gf = ceil_div(ns * 32, 256);
    if (gf > (int64_t)sm_count() * 32) gf = (int64_t)sm_count() * 32;
#define BSP_SELL_FILL(V, SC, D, PK)                                                                          \
  sell_fill_kernel<V, SC, D, PK><<<(unsigned)gf, 256, 0, s>>>(n, rowPtr, colIdx, P->val, P->slice_len,           \
                                                              P->slice_off, P->exps, (V *)P->lp_val, P->lp_cols)
    if (!mixed) {
      BSP_SELL_FILL(double, false, true, false);
    } else if (P->opt.mode == BSP_CG_MIXED_F32) {
      if (P->delta16) BSP_SELL_FILL(float, false, true, false); else BSP_SELL_FILL(float, false, false, false);
    } else if (P->opt.mode == BSP_CG_MIXED_F16) {
      if (P->delta16) BSP_SELL_FILL(__half, true, true, true); else BSP_SELL_FILL(__half, true, false, false);
    } else {
      if (P->delta16)
        BSP_SELL_FILL(__nv_bfloat16, true, true, true);
      else
        BSP_SELL_FILL(__nv_bfloat16, true, false, false);
    }
#undef BSP_SELL_FILL
    if (cudaGetLastError() != cudaSuccess) {
      set_error("bsp_cg_create: building the low-precision matrix failed");
      return BSP_ERR_CUDA;
    }
    *mat_bytes = padded * (packed ? 4 : (int64_t)vsz + (P->delta16 ? 2 : 4)) + (scaled ? (int64_t)n : 0) + 12 * ns;
  }
  return BSP_OK;
}
#undef BSP_CG_ALLOC

// Launch grids of the two kernels and the bytes counted per iteration.
static void plan_grids(bsp_cg_plan_s *P, int64_t mat_bytes) {
  const int32_t n = P->n;
  const bool mixed = cg_mixed(P);
  const int64_t vt = mixed ? 4 : 8;
  int oa = 4, ob = 4;  // partials were sized for the largest grid
  cg_plan_occupancy(P, oa, ob);
  P->grid_a = cg_grid(n, oa);
  P->grid = cg_grid(n, ob);
  // algorithmic bytes.  Two kernels: A reads the matrix, r and p_prev (own rows;
  // gathers counted once) and writes p and q; B reads p, q, x, r and writes x, r.
  // Preconditioned: the update kernel also reads M^{-1} and writes z.  Fused: the
  // diagonals and the published p (value and tag, written and read once) per
  // iteration, x, r and p in and out once per chunk; the rest stays on the SMs.
  if (P->fused_ctas) {
    P->bytes_iter = mat_bytes + 2 * (int64_t)fused_pub_bytes(P);
    P->bytes_chunk = 6 * vt * n;
  } else {
    P->bytes_chunk = 0;
    P->bytes_iter = mat_bytes + (mixed || P->sell64 ? 0 : 4 * ((int64_t)n + 1)) + 10 * vt * n;
    if (P->prec_bs)
      P->bytes_iter += vt * (ceil_div(n, P->prec_bs) * P->prec_bs * P->prec_bs + (int64_t)n);
  }
}

struct FusedLaunch {
  const void *kernel, *fill;
  int threads;
  size_t vsz;  // bytes of a stored value
};
template <typename V, typename VT, int THREADS>
static FusedLaunch fused_for(const bsp_cg_plan_s *P) {
  const int nd = P->fused_nd;
  const void *k;
  if (P->fused_polls < kFusedPolls)
    k = nd <= 5   ? (const void *)cg_fused_kernel<V, VT, 5, THREADS, true>
        : nd <= 7 ? (const void *)cg_fused_kernel<V, VT, 7, THREADS, true>
                  : (const void *)cg_fused_kernel<V, VT, 8, THREADS, true>;
  else
    k = nd <= 5   ? (const void *)cg_fused_kernel<V, VT, 5, THREADS, false>
        : nd <= 7 ? (const void *)cg_fused_kernel<V, VT, 7, THREADS, false>
                  : (const void *)cg_fused_kernel<V, VT, 8, THREADS, false>;
  return {k, (const void *)fused_fill_kernel<V, sizeof(V) == 2>, THREADS, sizeof(V)};
}

static FusedLaunch fused_launch(const bsp_cg_plan_s *P) {
  switch (P->opt.mode) {
    case BSP_CG_FP64: return fused_for<double, double, kFusedThreads64>(P);
    case BSP_CG_MIXED_F32: return fused_for<float, float, kFusedThreads32>(P);
    case BSP_CG_MIXED_F16: return fused_for<__half, float, kFusedThreads32>(P);
    default: return fused_for<__nv_bfloat16, float, kFusedThreads32>(P);
  }
}

// Lets the kernel have all the dynamic shared memory that its own leaves (*most).
static bsp_status fused_allow_smem(const void *kernel, int64_t *most) {
  int dev = 0, optin = 0;
  cudaFuncAttributes fa{};
  BSP_CUDA(cudaGetDevice(&dev));
  BSP_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  BSP_CUDA(cudaFuncGetAttributes(&fa, kernel));
  *most = optin - (int64_t)fa.sharedSizeBytes;
  BSP_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)*most));
  return BSP_OK;
}

static size_t fused_pub_bytes(const bsp_cg_plan_s *P) {  // value and tag, rows of whole slices
  return 2 * (cg_mixed(P) ? 4 : 8) * (size_t)ceil_div(P->n, 32) * 32;
}

// Slots and published elements without an epoch, epoch 0, no error: the state before
// the first launch, and after one that gave up (its epoch is not stored, so the next
// launch would take that run's slots and elements for its own).
static bsp_status fused_reset(bsp_cg_plan_s *P, cudaStream_t s) {
  BSP_CUDA(cudaMemsetAsync(P->slots, 0, 2 * kFusedMaxCtas * sizeof(CgSlot), s));
  BSP_CUDA(cudaMemsetAsync(P->pub, 0, fused_pub_bytes(P), s));
  BSP_CUDA(cudaMemsetAsync(P->sc + 8, 0, 2 * sizeof(double), s));
  return BSP_OK;
}

// Rows between which two kernels are the faster iteration.  Below them the fused one
// is few CTAs, so its two grid sums are short; above them the vectors' traffic
// decides.  In between the sums take most of an iteration of many CTAs, while two
// kernels still run as fast as they can be launched.  7-point Poisson (5-point
// Laplacian), us per iteration, fused / two kernels: FP64 24^3 7.4 / 7.6, 28^3 8.1 /
// 7.5, 32^3 8.7 / 7.5 (200^2 7.9 / 7.0), 48^3 9.7 / 8.9, 56^3 10.5 / 10.4, 64^3 11.3 /
// 11.9; FP32 32^3 8.5 / 8.7, 36^3 9.6 / 8.7, 48^3 9.9 / 9.5 (256^2 7.4 / 7.2), 52^3
// 10.0 / 10.7.  FP16 differs by 3% either way there (40^3 7.8 / 8.9) and stays fused.
// A launch of 2 iterations pays for loading and storing the vectors: FP16 16^3 17.4 / 17.0,
// 48^3 18.6 / 16.2, 64^3 20.7 / 20.0, 700^2 20.5 / 19.8, 100^3 27.0 / 29.1; from 4 on the
// two differ by 3%.
static bool two_kernels_faster(int mode, int32_t n, int check_every) {
  if (check_every < 4 && n < 600000) return true;
  switch (mode) {
    case BSP_CG_FP64: return n > 18000 && n < 180000;
    case BSP_CG_MIXED_F32: return n > 36000 && n < 120000;
    default: return false;
  }
}

// Sets up the fused iteration where it applies: no preconditioner, one CTA per
// SM whose share of the vectors fits in shared memory, strictly ascending columns
// in every row, and at most kFusedDiags distinct diagonals that the rows fill by
// 3/4 or more.
static bsp_status fused_setup(bsp_cg_plan_s *P, cudaStream_t s) {
  if (P->prec_bs || two_kernels_faster(P->opt.mode, P->n, P->opt.check_every)) return BSP_OK;
  const size_t vt = cg_mixed(P) ? 4 : 8;
  int dev = 0, coop = 0, optin = 0, sms = 0, occ = 0;
  BSP_CUDA(cudaGetDevice(&dev));
  BSP_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
  BSP_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  BSP_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int64_t ns = ceil_div(P->n, 32);
  const int threads = vt == 4 ? kFusedThreads32 : kFusedThreads64;
  // a slice per warp before another CTA joins the sums
  const int64_t ctas = std::min<int64_t>(ceil_div(ns, threads / 32), std::min(sms, kFusedMaxCtas));
  const int64_t smem = ceil_div(ns, ctas) * 32 * 4 * (int64_t)vt;
  if (!coop || smem > optin) return BSP_OK;
  int32_t *d_set = nullptr, h_set[kFusedDiags + 1];
  BSP_TRY(dalloc(&d_set, kFusedDiags + 1, s));
  for (int k = 0; k < kFusedDiags; ++k) h_set[k] = kNoDiag;
  h_set[kFusedDiags] = 0;
  BSP_CUDA(cudaMemcpyAsync(d_set, h_set, sizeof(h_set), cudaMemcpyHostToDevice, s));
  const unsigned gd = (unsigned)std::min<int64_t>(ceil_div(P->n, 256), (int64_t)sm_count() * 8);
  fused_diags_kernel<<<gd, 256, 0, s>>>(P->n, P->rowPtr, P->colIdx, d_set, d_set + kFusedDiags);
  BSP_LAUNCH_CHECK();
  BSP_CUDA(cudaMemcpyAsync(h_set, d_set, sizeof(h_set), cudaMemcpyDeviceToHost, s));
  BSP_CUDA(cudaStreamSynchronize(s));
  dfree(d_set, s);
  const int nd = (int)(std::find(h_set, h_set + kFusedDiags, kNoDiag) - h_set);
  if (h_set[kFusedDiags] || nd == 0 || 4 * (int64_t)P->nnz < 3 * (int64_t)nd * P->n) return BSP_OK;
  std::sort(h_set, h_set + nd);
  // ascending, padded to the kernel's number with zero diagonals of its own row
  // before the last one (their values are 0)
  const int padded_nd = nd <= 5 ? 5 : nd <= 7 ? 7 : 8;
  for (int k = 0; k < kFusedDiags; ++k) P->fused_diags.d[k] = 0;
  for (int k = 0; k < nd; ++k) P->fused_diags.d[k + 1 == nd ? padded_nd - 1 : k] = h_set[k];
  const auto range = std::minmax_element(P->fused_diags.d + 1, P->fused_diags.d + padded_nd - 1);
  P->fused_diags.lo = *range.first;
  P->fused_diags.hi = *range.second;
  P->fused_nd = nd;
  const FusedLaunch L = fused_launch(P);
  int64_t most = 0;
  BSP_TRY(fused_allow_smem(L.kernel, &most));
  if (smem > most) return BSP_OK;
  BSP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, L.kernel, threads, (size_t)smem));
  if ((int64_t)occ * sms < ctas) return BSP_OK;
  // an optimisation: without room for its buffers the two kernels run
  if (pool_malloc(&P->fused_val, L.vsz * kFusedDiags * (size_t)ns * 32, s) != cudaSuccess ||
      pool_malloc(&P->pub, fused_pub_bytes(P), s) != cudaSuccess ||
      dalloc(&P->slots, 2 * kFusedMaxCtas, s) != BSP_OK) {
    cudaGetLastError();
    clear_error();
    if (P->fused_val) pool_free(P->fused_val, s);
    if (P->pub) pool_free(P->pub, s);
    P->fused_val = P->pub = nullptr;
    return BSP_OK;
  }
  BSP_TRY(fused_reset(P, s));
  const int64_t gf = std::min<int64_t>(ceil_div(P->n, 256), (int64_t)sm_count() * 32);
  void *args[] = {&P->n, &P->rowPtr, &P->colIdx, &P->val, &P->exps, &P->fused_diags, &P->fused_val};
  BSP_CUDA(cudaLaunchKernel(L.fill, dim3((unsigned)gf), dim3(256), args, 0, s));
  P->fused_ctas = (int)ctas;
  P->fused_smem = (size_t)smem;
  return BSP_OK;
}

static void fused_free(bsp_cg_plan_s *P, cudaStream_t s) {
  dfree(P->slots, s);
  if (P->pub) pool_free(P->pub, s);
  if (P->fused_val) pool_free(P->fused_val, s);
  P->pub = P->fused_val = nullptr;
  P->fused_ctas = 0;
}

// *fits: whether the launch was taken; a stream confined to some of the SMs (a green
// context's) has no room for all CTAs at once.
static bsp_status fused_chunk(bsp_cg_plan_s *P, cudaStream_t s, bool *fits) {
  const FusedLaunch L = fused_launch(P);
  int iters = P->opt.check_every, npart = P->grid;
  double *epoch = P->sc + 9, *err = P->sc + 8;
  void *args[] = {&P->n,   &P->fused_val, &P->fused_diags, &P->exps, &P->x,     &P->r,  &P->p[0], &P->pub,
                  &P->part_rr, &npart,    &P->sc,          &iters,   &P->slots, &epoch, &err, &P->fused_polls};
  // One fused launch at a time on a device, whatever the streams and threads:
  // two grids that wait for their own CTAs must not share the SMs by halves.
  static std::mutex turn;
  static std::map<unsigned long long, cudaEvent_t> last;  // by context
  std::lock_guard<std::mutex> lock(turn);
  cudaEvent_t &done = last[context_id()];
  if (done)
    BSP_CUDA(cudaStreamWaitEvent(s, done, 0));
  else
    BSP_CUDA(cudaEventCreateWithFlags(&done, cudaEventDisableTiming));
  const cudaError_t e =
      cudaLaunchCooperativeKernel(L.kernel, dim3(P->fused_ctas), dim3(L.threads), args, P->fused_smem, s);
  *fits = e != cudaErrorCooperativeLaunchTooLarge;
  if (!*fits) {
    cudaGetLastError();
    return BSP_OK;
  }
  BSP_CUDA(e);
  BSP_CUDA(cudaEventRecord(done, s));
  return BSP_OK;
}

static bsp_status cg_run_chunk(bsp_cg_plan_s *P, cudaStream_t s) {
  if (P->fused_ctas) {
    bool fits = false;
    BSP_TRY(fused_chunk(P, s, &fits));
    if (fits) return BSP_OK;
    // two kernels from here on: x, r, p and the scalars are where they start from
    int64_t mat_bytes = (int64_t)P->nnz * 12;
    fused_free(P, s);
    BSP_TRY(two_kernel_setup(P, s, &mat_bytes));
    plan_grids(P, mat_bytes);
  }
  if (!P->opt.use_graphs) return cg_chunk(P, s);
  if (!P->graph) {
    if (!P->graph_stream) BSP_CUDA(cudaStreamCreateWithFlags(&P->graph_stream, cudaStreamNonBlocking));
    cudaGraph_t graph = nullptr;
    BSP_CUDA(cudaStreamBeginCapture(P->graph_stream, cudaStreamCaptureModeThreadLocal));
    bsp_status st = cg_chunk(P, P->graph_stream);
    cudaError_t e = cudaStreamEndCapture(P->graph_stream, &graph);
    if (st != BSP_OK) return st;
    if (e != cudaSuccess) BSP_FAIL(BSP_ERR_CUDA, cudaGetErrorString(e));
    e = cudaGraphInstantiate(&P->graph, graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) BSP_FAIL(BSP_ERR_CUDA, cudaGetErrorString(e));
  }
  BSP_CUDA(cudaGraphLaunch(P->graph, s));
  return BSP_OK;
}

static bsp_status read_scalars(bsp_cg_plan_s *P, cudaStream_t s) {
  BSP_CUDA(cudaMemcpyAsync(P->h_sc, P->sc, kCgScalars * sizeof(double), cudaMemcpyDeviceToHost, s));
  BSP_CUDA(cudaStreamSynchronize(s));
  int32_t err = 0;
  memcpy(&err, P->h_sc + 8, sizeof(err));
  if (err) {
    BSP_TRY(fused_reset(P, s));
    BSP_FAIL(BSP_ERR_TIMEOUT, "a bounded wait of the fused CG iteration gave up");
  }
  return BSP_OK;
}

// True FP64 residual of x64 -> sc[2]; the iterated residual (and its r.r
// partials for the next iteration) is replaced by it.
// measure_dev (mixed modes): also ||r_true - r_iterated||^2 -> sc[7].
static bsp_status cg_true_residual(bsp_cg_plan_s *P, const double *b, cudaStream_t s, bool measure_dev = false) {
  const int g = P->grid;
  const unsigned gr = (unsigned)ceil_div(P->n, kCgThreads);
  double *r = cg_mixed(P) ? P->r64 : (double *)P->r;
  cg_residual_kernel<<<gr, kCgThreads, 0, s>>>(P->n, P->rowPtr, P->colIdx, P->val, b, P->x64, r);
  if (cg_mixed(P))
    cg_norm_kernel<float><<<g, kCgThreads, 0, s>>>(P->n, r, (float *)P->r, P->part_res, P->part_rr,
                                                    measure_dev ? P->part_zq : nullptr);
  else
    cg_norm_kernel<double><<<g, kCgThreads, 0, s>>>(P->n, r, nullptr, P->part_res, nullptr);
  BSP_LAUNCH_CHECK();
  if (!cg_mixed(P)) {  // the FP64 residual is the iterated one
    BSP_CUDA(cudaMemcpyAsync(P->part_rr, P->part_res, sizeof(double) * g, cudaMemcpyDeviceToDevice, s));
  }
  sum_partials_kernel<<<1, kCgThreads, 0, s>>>(P->part_res, g, P->sc + 2);
  BSP_LAUNCH_CHECK();
  if (measure_dev && cg_mixed(P)) {
    sum_partials_kernel<<<1, kCgThreads, 0, s>>>(P->part_zq, g, P->sc + 7);
    BSP_LAUNCH_CHECK();
  }
  if (P->prec_bs) {
    if (cg_mixed(P))
      launch_prec<float>(P, s);
    else
      launch_prec<double>(P, s);
    BSP_LAUNCH_CHECK();
  }
  return BSP_OK;
}

// M^{-1} (Jacobi or block-Jacobi) of the CSR matrix in the iteration precision.
template <typename VT>
static bsp_status build_minv(bsp_cg_plan_s *P, cudaStream_t s) {
  const int bs = P->prec_bs;
  const int64_t nb = ((int64_t)P->n + bs - 1) / bs;
  BSP_CUDA(pool_malloc(reinterpret_cast<void **>(&P->minv), sizeof(VT) * (size_t)(nb * bs * bs), s));
  int32_t *bad = nullptr;
  BSP_TRY(dalloc(&bad, 1, s));
  BSP_CUDA(cudaMemsetAsync(bad, 0, sizeof(int32_t), s));
  const unsigned gr = (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(nb, 128), (int64_t)sm_count() * 16));
  VT *mi = (VT *)P->minv;
  if (bs == 1)
    cg_minv_kernel<VT, 1><<<gr, 128, 0, s>>>(P->n, P->rowPtr, P->colIdx, P->val, mi, bad);
  else if (bs == 4)
    cg_minv_kernel<VT, 4><<<gr, 128, 0, s>>>(P->n, P->rowPtr, P->colIdx, P->val, mi, bad);
  else
    cg_minv_kernel<VT, 8><<<gr, 128, 0, s>>>(P->n, P->rowPtr, P->colIdx, P->val, mi, bad);
  BSP_LAUNCH_CHECK();
  int32_t h_bad = 0;
  const bsp_status st = read_i32(bad, &h_bad, s);
  dfree(bad, s);
  BSP_TRY(st);
  if (h_bad)
    BSP_FAIL(BSP_ERR_INVALID, bs == 1 ? "a diagonal entry is zero or not finite"
                                      : "a diagonal block is singular or not finite");
  return BSP_OK;
}

// Enters the flexible outer iteration from a folded state (x_lp = 0, r64 and
// r_lp = b - A x64): no previous direction, inner direction restarted.
static bsp_status fcg_begin(bsp_cg_plan_s *P, cudaStream_t s) {
  BSP_CUDA(cudaMemsetAsync(P->p64, 0, sizeof(double) * P->n, s));
  BSP_CUDA(cudaMemsetAsync(P->q64, 0, sizeof(double) * P->n, s));
  BSP_CUDA(cudaMemsetAsync(P->sc, 0, 2 * sizeof(double), s));
  BSP_CUDA(cudaMemsetAsync(P->sc + 5, 0, sizeof(double), s));
  return BSP_OK;
}

// One outer step with z = the inner solution since the last step; then the
// inner iteration restarts on the new residual.  ||r64||^2 -> sc[6].
static bsp_status fcg_step(bsp_cg_plan_s *P, cudaStream_t s) {
  const int g = P->grid;
  fcg_z_kernel<<<g, kCgThreads, 0, s>>>(P->n, (float *)P->x, P->z64, P->q64, P->part_zq);
  fcg_dir_kernel<<<g, kCgThreads, 0, s>>>(P->n, P->part_zq, g, P->sc + 5, P->z64, P->p64);
  fcg_spmv_kernel<<<g, kCgThreads, 0, s>>>(P->n, P->rowPtr, P->colIdx, P->val, P->p64, P->q64, P->r64,
                                           P->part_pq, P->part_pr);
  fcg_update_kernel<<<g, kCgThreads, 0, s>>>(P->n, P->part_pq, P->part_pr, g, P->sc + 5, P->x64, P->r64, P->p64,
                                             P->q64, (float *)P->r, P->part_res, P->part_rr);
  BSP_LAUNCH_CHECK();
  sum_partials_kernel<<<1, kCgThreads, 0, s>>>(P->part_res, g, P->sc + 6);
  BSP_LAUNCH_CHECK();
  BSP_CUDA(cudaMemsetAsync(P->sc, 0, 2 * sizeof(double), s));  // inner restart: beta = 0
  if (P->prec_bs) {
    launch_prec<float>(P, s);
    BSP_LAUNCH_CHECK();
  }
  return BSP_OK;
}

}  // namespace bsp

using namespace bsp;

extern "C" bsp_status bsp_cg_default_options(bsp_cg_options *o) {
  clear_error();
  BSP_CHECK_ARG(o, "null options");
  o->mode = BSP_CG_MIXED_F16;
  o->tol = 1e-10;
  o->max_iters = 20000;
  o->check_every = 16;
  o->reliable_delta = 0.1;
  o->use_graphs = 1;
  o->precond = BSP_CG_PRECOND_NONE;
  o->precond_block = 4;
  o->refine = BSP_CG_REFINE_AUTO;
  return BSP_OK;
}

extern "C" bsp_status bsp_cg_destroy(bsp_cg_plan P) {
  clear_error();
  if (!P) return BSP_OK;
  cudaStream_t s = 0;
  if (P->graph) cudaGraphExecDestroy(P->graph);
  if (P->graph_stream) cudaStreamDestroy(P->graph_stream);
  if (P->x == P->x64) P->x = nullptr;  // FP64 mode iterates on x64 itself
  dfree(P->x64, s);
  dfree(P->r64, s);
  for (void *v : {P->x, P->r, P->p[0], P->p[1], P->q, P->lp_val, P->z, P->minv})
    if (v) pool_free(v, s);
  dfree(P->part_rz, s);
  dfree(P->p64, s);
  dfree(P->q64, s);
  dfree(P->z64, s);
  dfree(P->part_zq, s);
  dfree(P->part_pr, s);
  fused_free(P, s);
  if (P->lp_cols) pool_free(P->lp_cols, s);
  dfree(P->exps, s);
  dfree(P->slice_len, s);
  dfree(P->slice_off, s);
  dfree(P->part_pq, s);
  dfree(P->part_rr, s);
  dfree(P->part_res, s);
  dfree(P->sc, s);
  if (P->h_sc) cudaFreeHost(P->h_sc);
  cudaStreamSynchronize(s);
  delete P;
  return BSP_OK;
}

extern "C" bsp_status bsp_cg_create(int32_t n, int32_t nnz, const int32_t *rowPtr, const int32_t *colIdx,
                                    const double *values, const bsp_cg_options *opt, bsp_cg_plan *out,
                                    bsp_stream_t stream) {
  clear_error();
  BSP_CHECK_ARG(out && opt, "null argument");
  BSP_CHECK_ARG(n > 0 && nnz >= 0 && rowPtr && colIdx && values, "bad matrix");
  BSP_CHECK_ARG(opt->mode >= BSP_CG_FP64 && opt->mode <= BSP_CG_MIXED_BF16, "unknown mode");
  BSP_CHECK_ARG(opt->tol > 0 && opt->check_every >= 1 && opt->max_iters >= 1, "bad options");
  BSP_CHECK_ARG(opt->reliable_delta > 0 && opt->reliable_delta < 1, "reliable_delta must be in (0, 1)");
  BSP_CHECK_ARG(opt->precond >= BSP_CG_PRECOND_NONE && opt->precond <= BSP_CG_PRECOND_BLOCK_JACOBI,
                "unknown preconditioner");
  BSP_CHECK_ARG(opt->precond != BSP_CG_PRECOND_BLOCK_JACOBI || opt->precond_block == 4 || opt->precond_block == 8,
                "precond_block must be 4 or 8");
  BSP_CHECK_ARG(opt->refine >= BSP_CG_REFINE_AUTO && opt->refine <= BSP_CG_REFINE_FLEXIBLE, "unknown refine");
  cudaStream_t s = as_stream(stream);
  bsp_cg_plan_s *P = new bsp_cg_plan_s();
  P->n = n;
  P->nnz = nnz;
  P->opt = *opt;
  P->opt.check_every += P->opt.check_every & 1;  // even: iteration parity restarts at every chunk
  P->rowPtr = rowPtr;
  P->colIdx = colIdx;
  P->val = values;
  P->grid = (int)std::min<int64_t>(ceil_div(n, kCgThreads), (int64_t)sm_count() * kCgMaxCtasPerSm);
  const bool mixed = cg_mixed(P);
  const size_t vt = mixed ? 4 : 8;
  bsp_status st = BSP_OK;
  auto fail = [&](bsp_status e) {
    bsp_cg_destroy(P);
    return e;
  };
#define BSP_CG_TRY(x)                         \
  do {                                        \
    if ((st = (x)) != BSP_OK) return fail(st); \
  } while (0)
#define BSP_CG_CUDA(x)                                                              \
  do {                                                                              \
    cudaError_t e_ = (x);                                                           \
    if (e_ != cudaSuccess) {                                                        \
      set_error(std::string("bsp_cg_create: ") + #x + " -> " + cudaGetErrorString(e_)); \
      return fail(BSP_ERR_ALLOC);                                                   \
    }                                                                               \
  } while (0)
  BSP_CG_TRY(dalloc(&P->x64, (size_t)n, s));
  BSP_CG_TRY(dalloc(&P->part_pq, (size_t)P->grid, s));
  BSP_CG_TRY(dalloc(&P->part_rr, (size_t)P->grid, s));
  BSP_CG_TRY(dalloc(&P->part_res, (size_t)P->grid, s));
  BSP_CG_TRY(dalloc(&P->sc, kCgScalars, s));
  BSP_CG_CUDA(cudaMemsetAsync(P->sc, 0, kCgScalars * sizeof(double), s));
  BSP_CG_CUDA(cudaMallocHost(reinterpret_cast<void **>(&P->h_sc), kCgScalars * sizeof(double)));
  if (mixed) {
    P->x = nullptr;  // x32 allocated below
  }
  for (void **v : {&P->x, &P->r, &P->p[0], &P->p[1], &P->q}) BSP_CG_CUDA(pool_malloc(reinterpret_cast<void **>(v), vt * (size_t)n, s));
  if (!mixed) {  // lanes per row from the mean row length
    const double mean = (double)nnz / n;
    P->lpr = mean <= 10.0 ? 1 : mean <= 20.0 ? 2 : mean <= 40.0 ? 4 : 8;
  }
  P->prec_bs = opt->precond == BSP_CG_PRECOND_JACOBI ? 1
               : opt->precond == BSP_CG_PRECOND_BLOCK_JACOBI ? opt->precond_block : 0;
  if (mixed) {
    BSP_CG_TRY(dalloc(&P->r64, (size_t)n, s));
    BSP_CG_TRY(dalloc(&P->p64, (size_t)n, s));
    BSP_CG_TRY(dalloc(&P->q64, (size_t)n, s));
    BSP_CG_TRY(dalloc(&P->z64, (size_t)n, s));
    BSP_CG_TRY(dalloc(&P->part_zq, (size_t)P->grid, s));
    BSP_CG_TRY(dalloc(&P->part_pr, (size_t)P->grid, s));
  }
  if (P->prec_bs) {
    BSP_CG_CUDA(pool_malloc(reinterpret_cast<void **>(&P->z), vt * (size_t)n, s));
    BSP_CG_TRY(dalloc(&P->part_rz, (size_t)P->grid, s));
    BSP_CG_TRY(mixed ? build_minv<float>(P, s) : build_minv<double>(P, s));
  }
  if (!mixed) {  // FP64 mode iterates directly on x64
    pool_free(P->x, s);
    P->x = P->x64;
  }
  int64_t mat_bytes = (int64_t)nnz * 12;
  // FP64 mode with short rows: an FP64 SELL-32 copy with 16-bit column
  // offsets (10 bytes per entry, coalesced, no row pointers) replaces the CSR
  // walk when its slices are uniform; otherwise the CSR kernel runs.
  const bool try64 = !mixed && P->lpr == 1;
  int64_t padded = 0;
  if (mixed || try64) {
    if (mixed && opt->mode != BSP_CG_MIXED_F32) {
      BSP_CG_TRY(dalloc(&P->exps, (size_t)n, s));
      const unsigned ge = (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(n, 256), (int64_t)sm_count() * 16));
      row_exp_kernel<<<ge, 256, 0, s>>>(n, rowPtr, values, P->exps);
    }
    BSP_CG_TRY(fused_setup(P, s));
  }
  if (P->fused_ctas) {  // the diagonals replace the SELL copy
    const int64_t vsz = !mixed ? 8 : opt->mode == BSP_CG_MIXED_F32 ? 4 : 2;
    mat_bytes = ceil_div(n, 32) * 32 * kFusedDiags * vsz + (P->exps ? (int64_t)n : 0);
    const int32_t *d = P->fused_diags.d;
    P->delta16 = std::all_of(d, d + kFusedDiags, [](int32_t v) { return v >= -32768 && v <= 32767; });
  } else {
    BSP_CG_TRY(two_kernel_setup(P, s, &mat_bytes));
  }
  plan_grids(P, mat_bytes);
#undef BSP_CG_TRY
#undef BSP_CG_CUDA
  P->bytes_residual = (int64_t)nnz * 12 + 4 * ((int64_t)n + 1) + 3 * 8 * (int64_t)n;
  // flexible outer step: F1 8n+8n+8n, F2 24n, F3 matrix + 4(n+1) + 32n, F4 52n
  P->bytes_outer = (int64_t)nnz * 12 + 4 * ((int64_t)n + 1) + 132 * (int64_t)n;
  if (cudaStreamSynchronize(s) != cudaSuccess) {
    set_error("bsp_cg_create: preparing the matrix failed");
    return fail(BSP_ERR_CUDA);
  }
  *out = P;
  return BSP_OK;
}

namespace bsp {
void cg_plan_view(const bsp_cg_plan_s *P, CgPlanView *v) {
  v->n = P->n;
  v->nnz = P->nnz;
  v->rowPtr = P->rowPtr;
  v->colIdx = P->colIdx;
  v->val = P->val;
  v->mixed = cg_mixed(P);
  v->prec_bs = P->prec_bs;
  v->minv = P->minv;
  v->check_every = P->opt.check_every;
  v->max_iters = P->opt.max_iters;
  v->tol = P->opt.tol;
}
}  // namespace bsp

extern "C" bsp_status bsp_cg_fused_ctas(bsp_cg_plan P, int32_t *ctas) {
  clear_error();
  BSP_CHECK_ARG(P && ctas, "null argument");
  *ctas = P->fused_ctas;
  return BSP_OK;
}

extern "C" bsp_status bsp_cg_set_wait_limit(bsp_cg_plan P, uint32_t polls) {
  clear_error();
  BSP_CHECK_ARG(P && polls > 0, "null plan or a limit of 0");
  P->fused_polls = polls;
  int64_t most = 0;
  return P->fused_ctas ? fused_allow_smem(fused_launch(P).kernel, &most) : BSP_OK;
}

extern "C" bsp_status bsp_cg_solve(bsp_cg_plan P, const double *b, double *x, bsp_cg_result *res,
                                   bsp_stream_t stream) {
  clear_error();
  BSP_CHECK_ARG(P && b && x && res, "null argument");
  cudaStream_t s = as_stream(stream);
  *res = bsp_cg_result{};
  const int g = P->grid;
  const bool mixed = cg_mixed(P);
  const size_t vt = mixed ? 4 : 8;
  struct Events {  // destroyed on every way out
    cudaEvent_t e[2] = {nullptr, nullptr};
    ~Events() {
      for (cudaEvent_t v : e)
        if (v) cudaEventDestroy(v);
    }
  } ev;
  cudaEvent_t &e0 = ev.e[0], &e1 = ev.e[1];
  BSP_CUDA(cudaEventCreate(&e0));
  BSP_CUDA(cudaEventCreate(&e1));
  BSP_CUDA(cudaEventRecord(e0, s));
  // ||b||^2, then x64 = x0
  cg_norm_kernel<double><<<g, kCgThreads, 0, s>>>(P->n, b, nullptr, P->part_res, nullptr);
  sum_partials_kernel<<<1, kCgThreads, 0, s>>>(P->part_res, g, P->sc + 3);
  BSP_LAUNCH_CHECK();
  BSP_CUDA(cudaMemcpyAsync(P->x64, x, sizeof(double) * P->n, cudaMemcpyDeviceToDevice, s));
  // start: iterated residual, p_prev = 0, rr_prev = 0 (beta_0 = 0)
  if (mixed) BSP_CUDA(cudaMemsetAsync(P->x, 0, vt * P->n, s));
  BSP_CUDA(cudaMemsetAsync(P->p[0], 0, vt * P->n, s));
  BSP_CUDA(cudaMemsetAsync(P->sc, 0, 2 * sizeof(double), s));
  BSP_TRY(cg_true_residual(P, b, s));
  BSP_TRY(read_scalars(P, s));
  const double bb = P->h_sc[3];
  const double target = P->opt.tol * P->opt.tol * bb;
  const double delta2 = P->opt.reliable_delta * P->opt.reliable_delta;
  double rmax2 = P->h_sc[2];
  int64_t residuals = 2, iters = 0;
  int32_t updates = 0, no_progress = 0;
  double best_true = P->h_sc[2];
  bool coarse = false;
  bool done = bb == 0.0 || P->h_sc[2] <= target;
  bool flex = mixed && P->opt.refine == BSP_CG_REFINE_FLEXIBLE;
  int32_t outer = 0;
  if (flex) BSP_TRY(fcg_begin(P, s));
  // replacements / outer steps that stop lowering the residual: the
  // low-precision copy is too coarse for this matrix
  auto progress = [&](double r2) {
    if (r2 < best_true) {
      best_true = r2;
      no_progress = 0;
    } else if (++no_progress >= kCgNoProgress) {
      coarse = true;
    }
  };
  int chunks = 0;  // since the last replacement / outer step
  while (!done && iters < P->opt.max_iters) {
    BSP_TRY(cg_run_chunk(P, s));
    iters += P->opt.check_every;
    ++chunks;
    BSP_TRY(read_scalars(P, s));
    const double rr = P->h_sc[4];
    const bool stalled = !(rr == rr);  // NaN
    const bool growing = mixed && (rr > kCgGrowth * rmax2 || chunks >= kCgInnerChunks);
    if (!(rr <= target || (mixed && rr <= delta2 * rmax2) || stalled || growing)) continue;
    chunks = 0;
    if (flex) {
      if (stalled) break;
      BSP_TRY(fcg_step(P, s));
      BSP_TRY(read_scalars(P, s));
      ++outer;
      double r2 = P->h_sc[6];
      if (r2 <= target) {  // confirm with the true residual (which also restarts the inner iteration)
        BSP_TRY(cg_true_residual(P, b, s));
        BSP_CUDA(cudaMemsetAsync(P->sc, 0, 2 * sizeof(double), s));
        BSP_TRY(read_scalars(P, s));
        ++residuals;
        r2 = P->h_sc[2];
      }
      rmax2 = r2;
      progress(r2);
      done = r2 <= target || coarse;
      continue;
    }
    // reliable update: fold the inner solution, replace the residual
    if (mixed) {
      cg_fold_kernel<float><<<g, kCgThreads, 0, s>>>(P->n, (float *)P->x, P->x64);
      BSP_LAUNCH_CHECK();
    }
    BSP_TRY(cg_true_residual(P, b, s, mixed));
    BSP_TRY(read_scalars(P, s));
    ++residuals;
    ++updates;
    // A true residual far (in direction, not only in norm) from the iterated
    // one it replaces: the low-precision matrix is far from A (a large
    // condition number times the storage rounding) and the kept direction no
    // longer fits the replaced residual.  AUTO switches to the flexible outer
    // iteration; RELIABLE restarts the direction (beta = 0, i.e. iterative
    // refinement with CG as the inner solver).
    if (mixed && (growing || P->h_sc[7] > kCgDeviation * kCgDeviation * rr)) {
      if (P->opt.refine == BSP_CG_REFINE_AUTO) {
        flex = true;
        BSP_TRY(fcg_begin(P, s));
      } else {
        BSP_CUDA(cudaMemsetAsync(P->sc, 0, 2 * sizeof(double), s));
      }
    }
    rmax2 = P->h_sc[2];
    progress(P->h_sc[2]);
    done = P->h_sc[2] <= target || stalled || coarse;
  }
  if (!done && mixed) {  // budget spent: apply what the inner solve has
    if (flex) {
      BSP_TRY(fcg_step(P, s));
      ++outer;
    } else {
      cg_fold_kernel<float><<<g, kCgThreads, 0, s>>>(P->n, (float *)P->x, P->x64);
      BSP_LAUNCH_CHECK();
    }
    BSP_TRY(cg_true_residual(P, b, s));
    ++residuals;
  }
  BSP_CUDA(cudaMemcpyAsync(x, P->x64, sizeof(double) * P->n, cudaMemcpyDeviceToDevice, s));
  BSP_CUDA(cudaEventRecord(e1, s));
  BSP_TRY(read_scalars(P, s));
  float ms = 0;
  cudaEventElapsedTime(&ms, e0, e1);
  res->iterations = (int32_t)iters;
  res->reliable_updates = updates;
  res->outer_steps = outer;
  res->seconds = ms * 1e-3;
  res->rel_residual = bb > 0 ? sqrt(P->h_sc[2] / bb) : 0.0;
  res->converged = res->rel_residual <= P->opt.tol;
  res->bytes_moved = residuals * P->bytes_residual + iters * P->bytes_iter +
                     iters / P->opt.check_every * P->bytes_chunk + (int64_t)outer * P->bytes_outer;
  res->delta16 = P->delta16 ? 1 : 0;
  if (!res->converged) {
    set_error("CG stopped at relative residual " + std::to_string(res->rel_residual) +
              (coarse ? ": the low-precision matrix is too coarse for this matrix's condition number "
                        "(residual replacements stopped reducing the residual); use mode f32 or fp64"
                      : ""));
    return BSP_ERR_NOT_CONVERGED;
  }
  return BSP_OK;
}
