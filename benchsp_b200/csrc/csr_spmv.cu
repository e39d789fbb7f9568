// CSR SpMV kernels for sm_100a.
//
// Replaces the reference's CSR paths:
//   spmv_fp64 (thread per row)            src/csrspmv.cu:39-57
//   spmv_fp64_balance (16-nnz chunks, atomics) src/csrspmv.cu:84-102
//   spmv_fp16/fp64 + *_long (row split at 128 nnz) src/spmv.cu:13-107
// with three deterministic kernels (no atomics, each y element written by
// exactly one thread except the merge-path carry fix-up, which runs after):
//   * scalar: one thread per row, left-to-right sum with separately rounded
//     multiply and add -- bit-identical to ref_spmv_fp64 / ref_spmv_fp16
//     (src/ref.cpp:3-37) on the same inputs;
//   * vector: a power-of-two group of lanes per row, 8 entries per lane loaded
//     before their x gathers, shuffle reduction; long rows by a warp or the CTA;
//   * merge-path: every warp takes an equal share of (rows + nnz) merge
//     items, so power-law rows cost the same as short ones; warp-level
//     segmented scan plus a carry fix-up kernel over a small workspace.
#include <algorithm>
#include <type_traits>

#include "bsp_internal.cuh"

namespace bsp {

template <typename V> struct AccOf { using T = float; };
template <> struct AccOf<double> { using T = double; };

template <typename V> __device__ __forceinline__ typename AccOf<V>::T to_acc(V v);
template <> __device__ __forceinline__ double to_acc<double>(double v) { return v; }
template <> __device__ __forceinline__ float to_acc<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_acc<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float to_acc<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename V> __device__ __forceinline__ V from_acc(typename AccOf<V>::T v);
template <> __device__ __forceinline__ double from_acc<double>(double v) { return v; }
template <> __device__ __forceinline__ float from_acc<float>(float v) { return v; }
template <> __device__ __forceinline__ __half from_acc<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 from_acc<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }

template <typename V, typename A>
__device__ __forceinline__ void store_y(V *y, int64_t i, A sum, A alpha, A beta) {
  A r = alpha * sum;
  if (beta != A(0)) r += beta * to_acc<V>(y[i]);
  y[i] = from_acc<V>(r);
}

// One thread per row, sum in column order with no fused multiply-add: the
// exact operation sequence of ref_spmv_fp64/ref_spmv_fp16 (src/ref.cpp).
template <typename V>
__global__ void __launch_bounds__(256) csr_scalar_kernel(int32_t rows, const int32_t *__restrict__ rowPtr,
                                                         const int32_t *__restrict__ colIdx,
                                                         const V *__restrict__ val, const V *__restrict__ x,
                                                         V *__restrict__ y, typename AccOf<V>::T alpha,
                                                         typename AccOf<V>::T beta) {
  using A = typename AccOf<V>::T;
  for (int32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x) {
    A sum = A(0);
    const int32_t e = rowPtr[r + 1];
    for (int32_t j = rowPtr[r]; j < e; ++j)
      sum = add_rn(sum, mul_rn(to_acc<V>(val[j]), to_acc<V>(__ldg(&x[colIdx[j]]))));
    if (alpha == A(1) && beta == A(0))
      y[r] = from_acc<V>(sum);
    else
      store_y<V, A>(y, r, sum, alpha, beta);
  }
}

constexpr int kCsrThreads = 256;
constexpr int kCsrWarps = kCsrThreads / 32;
constexpr int kWarpRowFactor = 16;
constexpr int kLongList = 64;
constexpr int kWarpCtas = 64;  // of csr_warp_kernel per SM, at most

// Positions among the nonzeros are of type J.  A step's loads lie up to kOvershoot
// entries behind a row's end before they are masked.  Where nnz leaves that much
// room below 2^31 J is int32_t, whose sums fold into the loads' offsets; otherwise
// uint32_t, which does not wrap (power-law 2^20, FP32 38.4 against 40.0 us; 10% of
// the rows of 600 among rows of 40, FP64 99.6 against 115.7).
constexpr int32_t kOvershoot = 8 * kCsrThreads;

// Sum of entries j, j + STRIDE, ... < e (U in flight), this thread's share of a row.
template <typename V, int STRIDE, int U, typename J>
__device__ __forceinline__ typename AccOf<V>::T strided_sum(J j, J e, const int32_t *__restrict__ colIdx,
                                                            const V *__restrict__ val, const V *__restrict__ x) {
  using A = typename AccOf<V>::T;
  A sum = A(0);
  for (; j < e; j += U * STRIDE) {
    int32_t c[U];
    V a[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool in = j + u * STRIDE < e;
      c[u] = in ? colIdx[j + u * STRIDE] : -1;
      a[u] = in ? val[j + u * STRIDE] : V(0);
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (c[u] >= 0) sum = fma(to_acc<V>(a[u]), to_acc<V>(__ldg(&x[c[u]])), sum);
  }
  return sum;
}

// A long row by the lane that holds it.  Not inlined: in line, sum_long_rows slows down
// (1M rows, Zipf 2.0, cap 1,000, FP32 44.8 -> 48.8 us).
template <typename V, typename J>
__device__ __noinline__ void sum_own_row(int64_t r, J s, J e, const int32_t *__restrict__ colIdx,
                                         const V *__restrict__ val, const V *__restrict__ x, V *__restrict__ y,
                                         typename AccOf<V>::T alpha, typename AccOf<V>::T beta) {
  store_y<V, typename AccOf<V>::T>(y, r, strided_sum<V, 1, 4>(s, e, colIdx, val, x), alpha, beta);
}

// Long rows are left out of the pass over a CTA's rows and summed after it by
// more threads: a warp per row up to kCtaRow entries, the whole CTA above
// (power-law rows: one 10,000-entry row was a chain of 78 dependent loads for
// the warp that met it).  With one lane per row, and no row above kOwnRow in the CTA,
// each lane sums its own: 2M rows, a tenth of them of 20 and the others empty, FP64
// 71 -> 40 us, FP16 58 -> 39 (without any list 33 and 25, but the power-law matrices
// below take 15 to 30% longer then).  A row's summation order depends on its length, on
// the matrix's mean and, up to kOwnRow, on whether its CTA has a longer one.
// CTAs without such rows pay one barrier.
//
// Sums the CTA's long rows: `mine` says that this thread holds one, row `r`
// with entries [s, e).  Every thread of the CTA calls it.
template <typename V, int LPR, typename J>
__device__ __forceinline__ void sum_long_rows(bool mine, int64_t r, int32_t s, int32_t e,
                                              const int32_t *__restrict__ rowPtr,
                                              const int32_t *__restrict__ colIdx, const V *__restrict__ val,
                                              const V *__restrict__ x, V *__restrict__ y,
                                              typename AccOf<V>::T alpha, typename AccOf<V>::T beta) {
  using A = typename AccOf<V>::T;
  // A CTA takes its rows above kCtaRow one after another, so where rows are long on
  // average (and several such rows share a CTA) the bound is higher: 10% of the rows
  // of 600 among rows of 40 (16 lanes), FP16 87 us at 512, 65 here.  With few lanes
  // 512 is the faster one: power-law 2^17 FP64 16.9 us, 18.4 at 1024; 2^14 11.4 at
  // 1024, 14.5 at 2048, 24.7 at 4096.
  constexpr int kCtaRow = LPR <= 4 ? 512 : LPR == 32 ? 0 : 128 * LPR;
  constexpr int kOwnRow = 64, kFar = 1 << 16;
  // loads in flight: 8 where they leave the pass over the rows its registers (with 8
  // in the other types it slows down: stencil 128^3 FP32 89 -> 91 us, FP64 130 -> 139)
  constexpr int U = sizeof(V) == 2 && LPR > 1 && LPR < 32 ? 8 : 4;
  struct LongRow {
    int32_t s, e, r;
  };
  __shared__ LongRow list[kLongList];
  __shared__ int32_t count[kCsrWarps];
  __shared__ A part[kCsrWarps];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (!__syncthreads_or(mine)) return;
  if (sizeof(A) == 8 && mine) {
    // read again rather than carried through the pass: with s and e alive the
    // FP64 kernel takes 40 registers, and 6 instead of 8 CTAs fit an SM
    asm volatile("ld.global.nc.s32 %0, [%1];" : "=r"(s) : "l"(rowPtr + r));
    asm volatile("ld.global.nc.s32 %0, [%1];" : "=r"(e) : "l"(rowPtr + r + 1));
  }
  const unsigned mask = __ballot_sync(0xffffffffu, mine);
  const bool far = LPR == 1 && __any_sync(0xffffffffu, mine && e - s > kOwnRow);
  if (lane == 0) count[w] = __popc(mask) + (far ? kFar : 0);
  __syncthreads();
  int32_t n = 0, base = 0;
#pragma unroll
  for (int q = 0; q < kCsrWarps; ++q) {
    base += q < w ? count[q] : 0;
    n += count[q];
  }
  if (LPR == 1 && n < kFar) {
    if (mine) sum_own_row<V, J>(r, (J)s, (J)e, colIdx, val, x, y, alpha, beta);
    return;
  }
  n %= kFar;
  base %= kFar;
  base += __popc(mask & ((1u << lane) - 1));
  for (int32_t first = 0; first < n; first += kLongList) {  // CTA-uniform
    const int32_t m = min(n - first, kLongList);
    __syncthreads();
    if (mine && base >= first && base < first + m) list[base - first] = {s, e, (int32_t)r};
    __syncthreads();
    for (int k = w; k < m && LPR < 32; k += kCsrWarps) {
      const LongRow L = list[k];
      if (L.e - L.s > kCtaRow) continue;
      const A sum = warp_sum(strided_sum<V, 32, U>((J)((J)L.s + lane), (J)L.e, colIdx, val, x));
      if (lane == 0) store_y<V, A>(y, L.r, sum, alpha, beta);
    }
    for (int k = 0; k < m; ++k) {
      const LongRow L = list[k];
      if (L.e - L.s <= kCtaRow) continue;
      const A sum = warp_sum(strided_sum<V, kCsrThreads, U>((J)((J)L.s + threadIdx.x), (J)L.e, colIdx, val, x));
      if (lane == 0) part[w] = sum;
      __syncthreads();
      if (threadIdx.x == 0) {
        A t = part[0];
        for (int h = 1; h < kCsrWarps; ++h) t += part[h];
        store_y<V, A>(y, L.r, t, alpha, beta);
      }
      __syncthreads();
    }
  }
}

// LPR lanes per row (LPR in {1,2,4,8,16}), one pass: the grid covers the rows.
//
// A warp's life is one chain (row pointers -> entries -> x -> y), so the bytes a
// lane has in flight set the rate: 8 entries per lane on half the lanes against
// 4, 27-point stencil 128^3: FP16 110 -> 76 us (floor 54), FP32 122 -> 90 (72),
// FP64 157 -> 130 (109); 16 per lane FP16 84, FP32 101, FP64 145.  No loop over
// passes (the grid was capped at 64 CTAs per SM): FP64 160 -> 141 us at 4 per
// lane.
//
// Rows of more than long_len entries are left to sum_long_rows (power-law 2^20,
// Zipf 2.0, cap 10k: FP64 119 -> 52 us, FP16 60 -> 39; 2^14 rows FP64 25 -> 9).
// long_len is kWarpRowFactor entries per lane, but no less than 4 times the mean:
// the barrier and the list only pay for rows far above the others.  2M rows of 7 on
// average with 5% of 17 to 24 (an unstructured mesh), FP16: 37.8 us, at 16 entries
// per lane alone 46.9 (FP32 44.2 against 51.8); power-law within 2% of it.  FP64 with
// one lane keeps 78 us there (73 without the list, which takes the registers that its
// later entries had).  No more than 64 per lane where a caller asks for few lanes (rows
// of 200, FP64, one lane: 152 -> 122 us).
//
// Resident CTAs: FP64 with several lanes needs 40 registers (6 CTAs; at 8 it
// spills, 138 us); FP64 with one lane is capped at 32 (at 40 the 1024 CTAs of a
// 512^2 grid take a second wave, 3.8 -> 4.5 us).
template <typename V, int LPR, int F, typename J>
__global__ void __launch_bounds__(kCsrThreads, LPR > 1 && sizeof(V) == 8 ? 6 : LPR > 1 || sizeof(V) == 8 ? 8 : 0)
    csr_vector_kernel(int32_t rows, const int32_t *__restrict__ rowPtr, const int32_t *__restrict__ colIdx,
                      const V *__restrict__ val, const V *__restrict__ x, V *__restrict__ y,
                      typename AccOf<V>::T alpha, typename AccOf<V>::T beta, int32_t long_len) {
  using A = typename AccOf<V>::T;
  const int sub = threadIdx.x & (LPR - 1);
  const int64_t r = (int64_t)blockIdx.x * (kCsrThreads / LPR) + threadIdx.x / LPR;
  const bool active = r < rows;
  const int32_t s = active ? rowPtr[r] : 0, e0 = active ? rowPtr[r + 1] : 0;
  const bool is_long = e0 - s > long_len;
  // Several lanes count positions from their own first entry, which leaves the
  // loads' offsets constant (rows of 30, FP16 53 -> 48 us; rows of 33, FP64 71 -> 66);
  // one lane, and FP32 (rows of 64 33 -> 31 us), count from the arrays' start.
  const int32_t left = is_long ? 0 : max(e0 - s - sub, 0);
  constexpr bool kOwn = LPR > 1 && sizeof(V) != 4;
  const J begin = kOwn ? 0 : (J)s + sub, end = begin + left;
  const int32_t *ci = kOwn ? colIdx + s + sub : colIdx;
  const V *va = kOwn ? val + s + sub : val;
  // The first F entries of each lane are loaded together, then their x
  // gathers together: the rowPtr -> column -> x chain is paid once per
  // F entries instead of once per entry.
  int32_t c[F];
  V a[F];
#pragma unroll
  for (int k = 0; k < F; ++k) {
    const J j = begin + k * LPR;
    c[k] = j < end ? ci[j] : -1;
    a[k] = j < end ? va[j] : V(0);
  }
  A sum = A(0);
#pragma unroll
  for (int k = 0; k < F; ++k)
    if (c[k] >= 0) sum = fma(to_acc<V>(a[k]), to_acc<V>(__ldg(&x[c[k]])), sum);
#pragma unroll 4
  for (J j = begin + F * LPR; j < end; j += LPR)
    sum = fma(to_acc<V>(va[j]), to_acc<V>(__ldg(&x[ci[j]])), sum);
#pragma unroll
  for (int o = LPR / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o, LPR);
  if (active && sub == 0 && !is_long) store_y<V, A>(y, r, sum, alpha, beta);
  sum_long_rows<V, LPR, J>(is_long && sub == 0, r, s, e0, rowPtr, colIdx, val, x, y, alpha, beta);
}

// The long rows of a CTA of csr_warp_kernel: its rows once more, a row per thread.  Not
// inlined, so that the pass over the rows keeps its registers.
template <typename V>
__device__ __noinline__ void sum_own_long_rows(int32_t rows, const int32_t *__restrict__ rowPtr,
                                               const int32_t *__restrict__ colIdx, const V *__restrict__ val,
                                               const V *__restrict__ x, V *__restrict__ y,
                                               typename AccOf<V>::T alpha, typename AccOf<V>::T beta,
                                               int32_t long_len) {
  const int64_t nwarps = (int64_t)gridDim.x * kCsrWarps;
  for (int64_t first = (int64_t)blockIdx.x * kCsrWarps; first < rows; first += 32 * nwarps) {  // CTA-uniform
    const int64_t r = first + (threadIdx.x & (kCsrWarps - 1)) + (threadIdx.x / kCsrWarps) * nwarps;
    const int32_t s = r < rows ? rowPtr[r] : 0, e = r < rows ? rowPtr[r + 1] : 0;
    sum_long_rows<V, 32, uint32_t>(e - s > long_len, r, s, e, rowPtr, colIdx, val, x, y, alpha, beta);
  }
}

// A warp per row (32 lanes), a warp taking several rows: long rows on average.  The list
// of csr_vector_kernel would take most rows here (60,000 rows of 600 near the diagonal,
// FP64 138 us, FP16 112; here 69 and 44), and a grid that covers the rows in one pass
// leaves a warp one chain long (200,000 rows of 200, FP64 102 us; here 84, at 4
// entries in flight 89).
//
// LIST: rows of more than long_len entries, 512 and 4 times the mean at least, are left
// to the CTA.  Where warps take several rows, a longer one holds back all that its CTA
// still has: 200,000 rows of 130 on average, the longest 20,000, FP64 391 -> 181 us.
// With a row per warp the list only costs (20,000 rows of 275, the longest 5,000, FP32
// 32 -> 37 us).
template <typename V, int F, bool LIST>
__global__ void __launch_bounds__(kCsrThreads) csr_warp_kernel(int32_t rows, const int32_t *__restrict__ rowPtr,
                                                               const int32_t *__restrict__ colIdx,
                                                               const V *__restrict__ val, const V *__restrict__ x,
                                                               V *__restrict__ y, typename AccOf<V>::T alpha,
                                                               typename AccOf<V>::T beta, int32_t long_len) {
  using A = typename AccOf<V>::T;
  const int lane = threadIdx.x & 31;
  const int64_t nwarps = (int64_t)gridDim.x * kCsrWarps;
  bool any_long = false;
  for (int64_t r = (int64_t)blockIdx.x * kCsrWarps + (threadIdx.x >> 5); r < rows; r += nwarps) {
    const int32_t s0 = rowPtr[r], e0 = rowPtr[r + 1];
    if (LIST && e0 - s0 > long_len) {  // warp-uniform
      any_long = true;
      continue;
    }
    const uint32_t s = (uint32_t)s0 + lane, e = e0;
    int32_t c[F];
    V a[F];
#pragma unroll
    for (int k = 0; k < F; ++k) {
      const uint32_t j = s + 32 * k;
      c[k] = j < e ? colIdx[j] : -1;
      a[k] = j < e ? val[j] : V(0);
    }
    A sum = A(0);
#pragma unroll
    for (int k = 0; k < F; ++k)
      if (c[k] >= 0) sum = fma(to_acc<V>(a[k]), to_acc<V>(__ldg(&x[c[k]])), sum);
#pragma unroll 4
    for (uint32_t j = s + 32 * F; j < e; j += 32)
      sum = fma(to_acc<V>(val[j]), to_acc<V>(__ldg(&x[colIdx[j]])), sum);
    sum = warp_sum(sum);
    if (lane == 0) store_y<V, A>(y, r, sum, alpha, beta);
  }
  if constexpr (LIST)
    if (__syncthreads_or(any_long)) sum_own_long_rows<V>(rows, rowPtr, colIdx, val, x, y, alpha, beta, long_len);
}

// Warp per 32 consecutive rows ("stream").  The warp's nonzero range
// [rowPtr[r0], rowPtr[r0+32]) is read in pieces of kStreamPiece entries:
// every lane loads kStreamPiece/32 values and column indices (one coalesced
// 256-byte access per array and step), issues their x gathers together and
// stores the products to shared memory; then each lane adds its own row's
// products of the piece left to right.  Every row costs the same dependent
// chain (rowPtr -> entries -> x) as in the thread-per-row kernel, but the
// entry loads are coalesced and all of a piece's gathers are in flight at
// once.  Multiply and add are rounded separately in column order, so the
// result equals csr_scalar_kernel's (and ref_spmv_fp64's) bit for bit.
constexpr int kStreamPiece = 256;
constexpr int kStreamThreads = 256;

// 48 registers (5 CTAs per SM).  Capped at 40 / 32 registers it measured
// 16.7 / 17.3 us against 16.5 us on the 7-point Poisson 64^3 (L2 flushed).
template <typename V>
__global__ void __launch_bounds__(kStreamThreads) csr_stream_kernel(int32_t rows, const int32_t *__restrict__ rowPtr,
                                                                    const int32_t *__restrict__ colIdx,
                                                                    const V *__restrict__ val,
                                                                    const V *__restrict__ x, V *__restrict__ y,
                                                                    typename AccOf<V>::T alpha,
                                                                    typename AccOf<V>::T beta) {
  using A = typename AccOf<V>::T;
  constexpr int K = kStreamPiece / 32;
  __shared__ A prod[kStreamThreads / 32][kStreamPiece];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  A *pw = prod[wib];
  const int64_t nblk = ((int64_t)rows + 31) / 32;
  const int64_t nwarps = (int64_t)gridDim.x * (kStreamThreads / 32);
  for (int64_t wb = (int64_t)blockIdx.x * (kStreamThreads / 32) + wib; wb < nblk; wb += nwarps) {
    const int64_t r = wb * 32 + lane;
    const bool active = r < rows;
    const int32_t rs = active ? rowPtr[r] : 0, re = active ? rowPtr[r + 1] : 0;
    const int32_t base = __shfl_sync(0xffffffffu, rs, 0);
    const int64_t last = min((int64_t)rows, wb * 32 + 32) - 1 - wb * 32;   // last active lane
    const int32_t end = __shfl_sync(0xffffffffu, re, (int)last);
    A sum = A(0);
    for (int32_t pb = base; pb < end; pb += kStreamPiece) {   // warp-uniform
      int32_t c[K];
      V a[K];
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const int32_t j = pb + k * 32 + lane;
        c[k] = j < end ? colIdx[j] : -1;
        a[k] = j < end ? val[j] : V(0);
      }
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (c[k] >= 0) pw[k * 32 + lane] = mul_rn(to_acc<V>(a[k]), to_acc<V>(__ldg(&x[c[k]])));
      __syncwarp();
      const int32_t lo = rs > pb ? rs : pb;
      const int32_t hi = re < pb + kStreamPiece ? re : pb + kStreamPiece;
      for (int32_t j = lo; j < hi; ++j) sum = add_rn(sum, pw[j - pb]);
      __syncwarp();
    }
    if (active) {
      if (alpha == A(1) && beta == A(0))
        y[r] = from_acc<V>(sum);
      else
        store_y<V, A>(y, r, sum, alpha, beta);
    }
  }
}

// ---------------------------------------------------------------------------
// Merge-path SpMV (FP64).  Merge items are the rows' end offsets
// (rowPtr[1..rows]) interleaved with the nnz indices 0..nnz-1; every thread
// consumes kItems consecutive items.  Path coordinate (i, j) = (rows
// finished, nnz consumed); a row-end item is taken before nnz item j when
// rowPtr[i+1] <= j.
constexpr int kMergeItems = 8;
constexpr int kMergeThreads = 256;
constexpr int kMergeWarpItems = kWarp * kMergeItems;

__device__ __forceinline__ void merge_path_search(int64_t diag, const int32_t *__restrict__ rowEnd,
                                                  int32_t rows, int32_t nnz, int32_t &i, int32_t &j) {
  int64_t lo = diag - nnz > 0 ? diag - nnz : 0;
  int64_t hi = diag < rows ? diag : rows;
  while (lo < hi) {
    int64_t mid = (lo + hi) >> 1;
    if ((int64_t)rowEnd[mid] <= diag - mid - 1)
      lo = mid + 1;
    else
      hi = mid;
  }
  i = (int32_t)lo;
  j = (int32_t)(diag - lo);
}

// Per-warp carry: the partial sum of the row a warp's range ends inside.
// carry_row = -1 when the warp ends exactly on a row boundary.
__global__ void __launch_bounds__(kMergeThreads) csr_merge_kernel(
    int32_t rows, int32_t nnz, const int32_t *__restrict__ rowPtr, const int32_t *__restrict__ colIdx,
    const double *__restrict__ val, const double *__restrict__ x, double *__restrict__ y, double alpha,
    double beta, int32_t *__restrict__ carry_row, double *__restrict__ carry_val) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * kMergeThreads + threadIdx.x) >> 5;
  const int64_t total = (int64_t)rows + nnz;
  const int64_t warp_begin = warp * kMergeWarpItems;
  if (warp_begin >= total) return;  // whole warp exits together
  const int64_t diag = warp_begin + (int64_t)lane * kMergeItems;
  const int64_t diag_end = diag + kMergeItems < total ? diag + kMergeItems : total;

  int32_t i = 0, j = 0;
  if (diag < total) merge_path_search(diag, rowPtr + 1, rows, nnz, i, j);

  double acc = 0.0;
  int32_t first_row = -1;  // first row that ends in this lane's range
  double first_val = 0.0;
  for (int64_t d = diag; d < diag_end; ++d) {
    if (i < rows && rowPtr[i + 1] <= j) {
      if (first_row < 0) {
        first_row = i;
        first_val = acc;
      } else {
        double r = alpha * acc;
        if (beta != 0.0) r += beta * y[i];
        y[i] = r;
      }
      acc = 0.0;
      ++i;
    } else {
      acc = fma(val[j], __ldg(&x[colIdx[j]]), acc);
      ++j;
    }
  }
  // Segmented inclusive scan of the lanes' trailing partials: a lane that
  // finished a row starts a new segment.
  const bool head = first_row >= 0;
  double seg = acc;
  bool seg_head = head;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    double v = __shfl_up_sync(0xffffffffu, seg, o);
    bool h = __shfl_up_sync(0xffffffffu, seg_head, o);
    if (lane >= o && !seg_head) {
      seg += v;
      seg_head = h;
    }
  }
  // carry_in for this lane = inclusive result of lane-1.
  double carry_in = __shfl_up_sync(0xffffffffu, seg, 1);
  if (lane == 0) carry_in = 0.0;
  if (head) {
    double r = alpha * (first_val + carry_in);
    if (beta != 0.0) r += beta * y[first_row];
    y[first_row] = r;
  }
  if (lane == 31) {
    // Row the warp ends inside (i after the last lane's items), if unfinished.
    const int64_t wend = warp_begin + kMergeWarpItems < total ? warp_begin + kMergeWarpItems : total;
    int32_t ei, ej;
    merge_path_search(wend, rowPtr + 1, rows, nnz, ei, ej);
    const bool open = ei < rows && ej > rowPtr[ei];
    carry_row[warp] = open ? ei : -1;
    carry_val[warp] = open ? seg : 0.0;
  }
}

// Adds the carries to the rows they belong to.  Carries are ordered by row;
// the first carry of each run of equal rows sums the run (deterministic).
__global__ void csr_merge_fixup_kernel(int64_t nwarps, const int32_t *__restrict__ carry_row,
                                       const double *__restrict__ carry_val, double *__restrict__ y,
                                       double alpha) {
  for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < nwarps;
       w += (int64_t)gridDim.x * blockDim.x) {
    const int32_t r = carry_row[w];
    if (r < 0) continue;
    if (w > 0 && carry_row[w - 1] == r) continue;
    double s = 0.0;
    for (int64_t k = w; k < nwarps && carry_row[k] == r; ++k) s += carry_val[k];
    y[r] += alpha * s;
  }
}

static int64_t merge_warps(int32_t rows, int32_t nnz) {
  return ceil_div((int64_t)rows + nnz, kMergeWarpItems);
}

bsp_status launch_merge(int32_t rows, int32_t nnz, const int32_t *rowPtr, const int32_t *colIdx,
                        const double *val, const double *x, double *y, double alpha, double beta,
                        int32_t *carry_row, double *carry_val, cudaStream_t s) {
  const int64_t nw = merge_warps(rows, nnz);
  if (nw == 0) return BSP_OK;
  const int64_t blocks = ceil_div(nw * kWarp, kMergeThreads);
  csr_merge_kernel<<<(unsigned)blocks, kMergeThreads, 0, s>>>(rows, nnz, rowPtr, colIdx, val, x, y, alpha,
                                                              beta, carry_row, carry_val);
  BSP_LAUNCH_CHECK();
  const int64_t fb = ceil_div(nw, 256);
  csr_merge_fixup_kernel<<<(unsigned)(fb < 4096 ? fb : 4096), 256, 0, s>>>(nw, carry_row, carry_val, y, alpha);
  BSP_LAUNCH_CHECK();
  return BSP_OK;
}

size_t merge_workspace_bytes(int32_t rows, int32_t nnz) {
  const int64_t nw = merge_warps(rows, nnz);
  const size_t rows_b = ((size_t)nw * sizeof(int32_t) + 255) & ~size_t(255);
  return rows_b + (size_t)nw * sizeof(double);
}

// ---------------------------------------------------------------------------
template <typename V, int F, typename J>
static void launch_lanes(int lpr, int32_t rows, int32_t long_len, const int32_t *rp, const int32_t *ci, const V *v,
                         const V *x, V *y, typename AccOf<V>::T a, typename AccOf<V>::T b, cudaStream_t s) {
  const unsigned blocks = (unsigned)ceil_div(rows, kCsrThreads / lpr);  // rows > 0
  switch (lpr) {
#define BSP_VEC_CASE(L)                                                                                   \
  case L:                                                                                                 \
    csr_vector_kernel<V, L, F, J><<<blocks, kCsrThreads, 0, s>>>(rows, rp, ci, v, x, y, a, b, long_len); \
    break;
    BSP_VEC_CASE(2) BSP_VEC_CASE(4) BSP_VEC_CASE(8) BSP_VEC_CASE(16)
#undef BSP_VEC_CASE
    case 1: csr_vector_kernel<V, 1, 8, J><<<blocks, kCsrThreads, 0, s>>>(rows, rp, ci, v, x, y, a, b, long_len); break;
    case 32:
      if (ceil_div(rows, kCsrWarps) > kWarpCtas * sm_count())
        csr_warp_kernel<V, F, true><<<kWarpCtas * sm_count(), kCsrThreads, 0, s>>>(rows, rp, ci, v, x, y, a, b, long_len);
      else
        csr_warp_kernel<V, 8, false><<<blocks, kCsrThreads, 0, s>>>(rows, rp, ci, v, x, y, a, b, 0);
      break;
  }
}

template <typename V>
static bsp_status launch_vector(int lpr, int32_t rows, int32_t nnz, const int32_t *rp, const int32_t *ci, const V *v,
                                const V *x, V *y, typename AccOf<V>::T a, typename AccOf<V>::T b,
                                cudaStream_t s) {
  if (lpr < 1 || lpr > 32 || (lpr & (lpr - 1)) != 0)
    BSP_FAIL(BSP_ERR_INVALID, "lanes_per_row must be a power of two in [1,32]");
  // fewer lanes than auto_lanes gives: the bound stays with the lanes
  const int64_t mean4 = 4 * (int64_t)nnz / rows;
  const int32_t long_len = (int32_t)std::min<int64_t>(
      INT32_MAX, std::max<int64_t>(kWarpRowFactor * lpr, lpr == 32 ? mean4 : std::min<int64_t>(64 * lpr, mean4)));
  // 4 entries per lane loaded together instead of 8 where rows do not fill those: asked
  // for more lanes than auto_lanes gives (rows of 5, FP64: 8 lanes 59 -> 53 us, 32 184
  // -> 151), or a warp per row (rows of 90 160 -> 135 us, of 160 even)
  const bool four = nnz <= 2ll * lpr * rows || nnz == 4ll * lpr * rows || (lpr == 32 && nnz <= 160ll * rows);
  const bool room = nnz <= INT32_MAX - kOvershoot;
  if (four && room)
    launch_lanes<V, 4, int32_t>(lpr, rows, long_len, rp, ci, v, x, y, a, b, s);
  else if (four)
    launch_lanes<V, 4, uint32_t>(lpr, rows, long_len, rp, ci, v, x, y, a, b, s);
  else if (room)
    launch_lanes<V, 8, int32_t>(lpr, rows, long_len, rp, ci, v, x, y, a, b, s);
  else
    launch_lanes<V, 8, uint32_t>(lpr, rows, long_len, rp, ci, v, x, y, a, b, s);
  BSP_LAUNCH_CHECK();
  return BSP_OK;
}

template <typename V>
static bsp_status launch_scalar(int32_t rows, const int32_t *rp, const int32_t *ci, const V *v, const V *x,
                                V *y, typename AccOf<V>::T a, typename AccOf<V>::T b, cudaStream_t s) {
  int64_t blocks = ceil_div(rows, 256);
  const int64_t cap = (int64_t)sm_count() * 64;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  csr_scalar_kernel<V><<<(unsigned)blocks, 256, 0, s>>>(rows, rp, ci, v, x, y, a, b);
  BSP_LAUNCH_CHECK();
  return BSP_OK;
}

template <typename V>
static bsp_status launch_stream(int32_t rows, const int32_t *rp, const int32_t *ci, const V *v, const V *x, V *y,
                                typename AccOf<V>::T a, typename AccOf<V>::T b, cudaStream_t s) {
  const int64_t warps = ceil_div(rows, 32);
  int64_t blocks = ceil_div(warps, kStreamThreads / 32);
  const int64_t cap = (int64_t)sm_count() * 32;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  csr_stream_kernel<V><<<(unsigned)blocks, kStreamThreads, 0, s>>>(rows, rp, ci, v, x, y, a, b);
  BSP_LAUNCH_CHECK();
  return BSP_OK;
}

// Lanes per row from the mean row length: the smallest power of two whose lanes
// hold the row in their 8 entries loaded together, up to 64 entries; a few more by the
// same lanes cost less than twice the lanes (rows of 70, 60M nonzeros, FP64: 8 lanes 131
// us, 16 177; rows of 130, FP16: 16 lanes 78, 32 107), and above that FP64 has a warp per
// row, 4 loaded together (rows of 90: 135 us, 16 lanes 146; of 160: 119 against 142).
// A mean of 16 (32) exactly is almost always rows of one length, whose starts then lie
// on the same banks of L1: twice the lanes with 4 entries each (rows of 16, 8M nonzeros:
// FP32 20.6 -> 14.5 us, FP16 16.6 -> 12.5, FP64 31 -> 25; of 32: FP32 20.4 -> 14.5, FP16
// 16.5 -> 12.5, FP64 24.7 and 23.2 but 144 and 160 at 60M).
int auto_lanes(int32_t rows, int32_t nnz, size_t value_bytes) {
  const double mean = rows > 0 ? (double)nnz / rows : 0.0;
  const bool wide = value_bytes == 8;
  if (mean == 16.0) return 4;
  if (mean == 32.0 && !wide) return 8;
  if (mean > 64.0) return wide ? (mean <= 88.0 ? 8 : 32) : (mean <= 144.0 ? 16 : 32);
  int l = 1;
  while (8.0 * l < mean) l <<= 1;
  return l;
}

template <typename V>
static bsp_status csr_dispatch(int32_t rows, int32_t nnz, const int32_t *rp, const int32_t *ci, const V *v,
                               const V *x, V *y, double alpha, double beta, int32_t algo, int32_t lpr,
                               cudaStream_t s) {
  using A = typename AccOf<V>::T;
  if (algo == BSP_CSR_SCALAR) return launch_scalar<V>(rows, rp, ci, v, x, y, (A)alpha, (A)beta, s);
  if (algo == BSP_CSR_STREAM) return launch_stream<V>(rows, rp, ci, v, x, y, (A)alpha, (A)beta, s);
  if (lpr <= 0) lpr = auto_lanes(rows, nnz, sizeof(V));
  return launch_vector<V>(lpr, rows, nnz, rp, ci, v, x, y, (A)alpha, (A)beta, s);
}

}  // namespace bsp

using namespace bsp;

extern "C" size_t bsp_csr_merge_workspace(int32_t rows, int32_t nnz) {
  return merge_workspace_bytes(rows, nnz);
}

extern "C" bsp_status bsp_csr_spmv_merge_f64(int32_t rows, int32_t cols, int32_t nnz, const int32_t *rowPtr,
                                             const int32_t *colIdx, const double *values, const double *x,
                                             double *y, double alpha, double beta, void *workspace,
                                             size_t workspace_bytes, bsp_stream_t stream) {
  clear_error();
  BSP_CHECK_ARG(rows >= 0 && cols >= 0 && nnz >= 0, "negative size");
  if (rows == 0) return BSP_OK;
  BSP_CHECK_ARG(rowPtr && y, "null pointer");
  BSP_CHECK_ARG(nnz == 0 || (colIdx && values && x), "null pointer");
  const size_t need = merge_workspace_bytes(rows, nnz);
  BSP_CHECK_ARG(workspace && workspace_bytes >= need, "workspace too small");
  BSP_CHECK_ARG(((uintptr_t)workspace & 15) == 0, "workspace must be 16-byte aligned");
  const int64_t nw = ceil_div((int64_t)rows + nnz, kMergeWarpItems);
  int32_t *carry_row = reinterpret_cast<int32_t *>(workspace);
  double *carry_val = reinterpret_cast<double *>(reinterpret_cast<char *>(workspace) +
                                                 (((size_t)nw * sizeof(int32_t) + 255) & ~size_t(255)));
  return launch_merge(rows, nnz, rowPtr, colIdx, values, x, y, alpha, beta, carry_row, carry_val,
                      as_stream(stream));
}

extern "C" bsp_status bsp_csr_spmv(int32_t rows, int32_t cols, int32_t nnz, const int32_t *rowPtr,
                                   const int32_t *colIdx, const void *values, bsp_dtype dtype, const void *x,
                                   void *y, double alpha, double beta, int32_t algo, int32_t lanes_per_row,
                                   bsp_stream_t stream) {
  clear_error();
  BSP_CHECK_ARG(rows >= 0 && cols >= 0 && nnz >= 0, "negative size");
  if (rows == 0) return BSP_OK;
  BSP_CHECK_ARG(rowPtr && y, "null pointer");
  BSP_CHECK_ARG(nnz == 0 || (colIdx && values && x), "null pointer");
  BSP_CHECK_ARG(lanes_per_row >= 0 && lanes_per_row <= 32 && (lanes_per_row & (lanes_per_row - 1)) == 0,
                "lanes_per_row must be 0 or a power of two <= 32");
  cudaStream_t s = as_stream(stream);
  if (algo == BSP_CSR_MERGE) {
    BSP_CHECK_ARG(dtype == BSP_F64, "merge-path is FP64 only");
    const size_t need = merge_workspace_bytes(rows, nnz);
    void *ws = nullptr;
    BSP_CUDA(pool_malloc(reinterpret_cast<void **>(&ws), need, s));
    bsp_status st = bsp_csr_spmv_merge_f64(rows, cols, nnz, rowPtr, colIdx, (const double *)values,
                                           (const double *)x, (double *)y, alpha, beta, ws, need, stream);
    pool_free(ws, s);
    return st;
  }
  if (algo == BSP_CSR_AUTO) {
    // Irregular rows (max far above mean) go through merge-path; the row
    // statistics are not known here without a pass, so AUTO means VECTOR
    // with lanes from the mean.  Plans pick MERGE from measured features.
    algo = BSP_CSR_VECTOR;
  }
  BSP_CHECK_ARG(algo == BSP_CSR_VECTOR || algo == BSP_CSR_SCALAR || algo == BSP_CSR_STREAM, "unknown algo");
  switch (dtype) {
    case BSP_F64:
      return csr_dispatch<double>(rows, nnz, rowPtr, colIdx, (const double *)values, (const double *)x,
                                  (double *)y, alpha, beta, algo, lanes_per_row, s);
    case BSP_F32:
      return csr_dispatch<float>(rows, nnz, rowPtr, colIdx, (const float *)values, (const float *)x,
                                 (float *)y, alpha, beta, algo, lanes_per_row, s);
    case BSP_F16:
      return csr_dispatch<__half>(rows, nnz, rowPtr, colIdx, (const __half *)values, (const __half *)x,
                                  (__half *)y, alpha, beta, algo, lanes_per_row, s);
    case BSP_BF16:
      return csr_dispatch<__nv_bfloat16>(rows, nnz, rowPtr, colIdx, (const __nv_bfloat16 *)values,
                                         (const __nv_bfloat16 *)x, (__nv_bfloat16 *)y, alpha, beta, algo,
                                         lanes_per_row, s);
  }
  BSP_FAIL(BSP_ERR_INVALID, "unknown dtype");
}
