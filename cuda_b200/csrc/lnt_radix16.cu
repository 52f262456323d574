// Two-pass squaring with register passes (smem_passes.cuh) for n = 2^13 ... 2^26.
//
// Same layout, twiddle tables and carry scheme as lnt_twopass.cu (which
// replaces the reference's FFT_2SMEM pool, kernel_pool.cu:39-48): columns of
// n2 words and rows of n1 words, transformed in shared memory; the result of
// the forward transform is in fully bit-reversed order, like the radix-2
// kernels, so all plans share the 4-step twiddle tables.
//
// row_square_r16: the first pass reads HBM directly (with the 4-step twiddle)
// and the last inverse pass writes HBM directly; the last forward pass, the
// pointwise square and the first inverse pass run in registers back to back.
#include <map>
#include <type_traits>
#include <mutex>
#include <utility>

#include "carry.cuh"
#include "lnt_internal.h"
#include "smem_passes.cuh"

namespace lnt {

namespace {

using namespace smem;

// ------------------------------------------------------------------ rows ----

// 256 threads per row of up to 4096 words (four CTAs per SM); longer rows hold
// one or two CTAs per SM, so their CTAs are wider to keep 32 warps per SM.
constexpr int row_threads_for(int L) { return L <= 4096 ? 256 : (L == 8192 ? 512 : 1024); }
// The squaring kernel's CTA for `rows` rows of L words: in a launch that fills
// the GPU, up to 4096 words take two radix-8 tasks per thread per pass (256
// threads for 4096 words, down to one warp); a launch of fewer CTAs than twice
// the SMs (latency) keeps 256; longer rows as row_threads_for.
constexpr int row_square_threads(int L, int rows, bool latency) {
  return L > 4096 ? row_threads_for(L)
                  : (L * rows >= 4096 || latency ? 256
                                                 : (L * rows >= 2048 ? 128 : (L * rows >= 1024 ? 64 : 32)));
}
// CTAs of TH threads an SM that the kernels are compiled for.  Passes of up to 8 points: 1024 threads,
// 64 registers.  Passes of 16 points hold 48 registers of three-word values and the twiddles: 512
// threads, 128 registers.  `Dense`: 768 threads, 80 registers; they spill (264 bytes in col_fused), which
// only a launch of many CTAs makes up for (col_dense).
template <int TH, int MR, bool Dense = false>
constexpr int min_blocks() {
  constexpr int threads = MR == 16 ? (Dense ? 768 : 512) : 1024;
  return threads / TH > 0 ? threads / TH : 1;
}

// Forward pass of `rows` row transforms.  The first pass (span = L) reads HBM
// and applies the 4-step twiddle; later passes read shared memory.  One code
// body serves both, which keeps the kernel small for the instruction cache.
template <int R, bool Big>
__device__ __forceinline__ void row_dif_tasks(uint64_t* sm, int ld, int rows, int L, int span,
                                              const uint64_t* x, const uint64_t* twf,
                                              const uint64_t* twL) {
  const bool first = span == L;
  const int q = span / R, per = L / R, qs = q + (q >> 4);
  const int lq = __ffs(q) - 1, lper = __ffs(per) - 1;
  for (int task = threadIdx.x; task < rows * per; task += blockDim.x) {
    const int g = task >> lper, k = swap_tasks<R>(task & (per - 1), q, per), b = k >> lq, t = k & (q - 1);
    const int off = b * span + t, b0 = sw(off);
    uint64_t* base = sm + g * ld;
    uint64_t v[R];
    lazy::W3 y[R];
    if (first) {
      const size_t rb = (size_t)g * L + off;
#pragma unroll
      for (int d = 0; d < R; ++d) y[d] = lazy::mul3(x[rb + q * d], twf[rb + q * d]);
    } else {
#pragma unroll
      for (int d = 0; d < R; ++d) y[d] = lazy::from_word(base[task_pos<Big>(b0, q, qs, d)]);
    }
    lazy::dif<R>(y, v);
    if (q > 1) mul_task_twiddles<R>(v, twL, t, q);
#pragma unroll
    for (int r = 0; r < R; ++r) base[task_pos<Big>(b0, q, qs, r)] = v[r];
  }
}

// Inverse pass; the last one (span = L) applies the inverse 4-step twiddle and
// writes HBM.
template <int R, bool Big>
__device__ __forceinline__ void row_dit_tasks(uint64_t* sm, int ld, int rows, int L, int span,
                                              uint64_t* x, const uint64_t* twi, const uint64_t* itwL) {
  const bool last = span == L;
  const int q = span / R, per = L / R, qs = q + (q >> 4);
  const int lq = __ffs(q) - 1, lper = __ffs(per) - 1;
  for (int task = threadIdx.x; task < rows * per; task += blockDim.x) {
    const int g = task >> lper, k = swap_tasks<R>(task & (per - 1), q, per), b = k >> lq, t = k & (q - 1);
    const int off = b * span + t, b0 = sw(off);
    uint64_t* base = sm + g * ld;
    uint64_t v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = base[task_pos<Big>(b0, q, qs, r)];
    lazy::W3 y[R];
    if (q > 1)
      mul_task_twiddles<R>(v, itwL, t, q, y);
    else
      widen<R>(v, y);
    lazy::dit_inv<R>(y, v);
    if (last) {
      const size_t rb = (size_t)g * L + off;
#pragma unroll
      for (int d = 0; d < R; ++d) x[rb + q * d] = lazy::mul(v[d], twi[rb + q * d]);
    } else {
#pragma unroll
      for (int d = 0; d < R; ++d) base[task_pos<Big>(b0, q, qs, d)] = v[d];
    }
  }
}

#ifndef LNT_ROW_STRIDED
#define LNT_ROW_STRIDED 1
#endif

template <int R>
__device__ void row_dif_pass(uint64_t* sm, int ld, int rows, int L, int span, const uint64_t* x,
                             const uint64_t* twf, const uint64_t* twL) {
  if (LNT_ROW_STRIDED && span / R >= 16)
    row_dif_tasks<R, true>(sm, ld, rows, L, span, x, twf, twL);
  else
    row_dif_tasks<R, false>(sm, ld, rows, L, span, x, twf, twL);
}

template <int R>
__device__ void row_dit_pass(uint64_t* sm, int ld, int rows, int L, int span, uint64_t* x,
                             const uint64_t* twi, const uint64_t* itwL) {
  if (LNT_ROW_STRIDED && span / R >= 16)
    row_dit_tasks<R, true>(sm, ld, rows, L, span, x, twi, itwL);
  else
    row_dit_tasks<R, false>(sm, ld, rows, L, span, x, twi, itwL);
}

template <bool Forward, int MR>
__device__ __forceinline__ void row_pass_r(int R, uint64_t* sm, int ld, int rows, int L, int span,
                                           uint64_t* x, const uint64_t* tw4, const uint64_t* twL) {
  switch (R) {
    case 2:
      if constexpr (Forward) row_dif_pass<2>(sm, ld, rows, L, span, x, tw4, twL);
      else row_dit_pass<2>(sm, ld, rows, L, span, x, tw4, twL);
      break;
    case 4:
      if constexpr (Forward) row_dif_pass<4>(sm, ld, rows, L, span, x, tw4, twL);
      else row_dit_pass<4>(sm, ld, rows, L, span, x, tw4, twL);
      break;
    case 8:
      if constexpr (Forward) row_dif_pass<8>(sm, ld, rows, L, span, x, tw4, twL);
      else row_dit_pass<8>(sm, ld, rows, L, span, x, tw4, twL);
      break;
    default:
      if constexpr (MR >= 16) {
        if constexpr (Forward) row_dif_pass<16>(sm, ld, rows, L, span, x, tw4, twL);
        else row_dit_pass<16>(sm, ld, rows, L, span, x, tw4, twL);
      }
      break;
  }
}

// the pass tables of a row of n1 words
template <int MR>
__device__ __forceinline__ const uint64_t* row_tw(const TwoPassDesc& D) { return MR == 16 ? D.itw1x : D.itw1; }
template <int MR>
__device__ __forceinline__ const uint64_t* row_itw(const TwoPassDesc& D) { return MR == 16 ? D.iitw1x : D.iitw1; }

template <int TH, int MR>
__global__ void __launch_bounds__(TH, min_blocks<TH, MR>()) row_square_r16(const TwoPassDesc* __restrict__ Ds, Passes P, int rows) {
  extern __shared__ __align__(16) uint64_t sm[];
  const TwoPassDesc& D = Ds[blockIdx.y];
  const int L = (int)D.n1, ld = padded(L);
  const size_t off = (size_t)blockIdx.x * rows * L;
  uint64_t* x = reinterpret_cast<uint64_t*>(D.x) + off;
  int span = L;
  for (int j = 0, seg = 0; j + 1 < P.m; ++j) {
    row_pass_r<true, MR>(P.radix[j], sm, ld, rows, L, span, x, D.twf + off, row_tw<MR>(D) + seg);
    seg += span;
    span /= P.radix[j];
    __syncthreads();
  }
  pass_r<2, MR>(P.radix[P.m - 1], sm, ld, rows, L, span, nullptr);
  __syncthreads();
  for (int j = P.m - 2; j >= 0; --j) {
    span *= P.radix[j];
    row_pass_r<false, MR>(P.radix[j], sm, ld, rows, L, span, x, D.twi + off,
                      row_itw<MR>(D) + pass_table_offset(P, L, j));
    if (j) __syncthreads();
  }
}

// Forward row transforms only (the first half of row_square_r16): the rows
// after all forward passes, in the order the passes leave them, go back to x.
// With col_forward before it this is the full transform of a residue, the
// operand of a product (row_mul_r16).
template <int TH, int MR>
__global__ void __launch_bounds__(TH) row_forward_r16(const TwoPassDesc* __restrict__ Ds, Passes P, int rows) {
  extern __shared__ __align__(16) uint64_t sm[];
  const TwoPassDesc& D = Ds[blockIdx.y];
  const int L = (int)D.n1, ld = padded(L);
  const size_t off = (size_t)blockIdx.x * rows * L;
  uint64_t* x = reinterpret_cast<uint64_t*>(D.x) + off;
  int span = L;
  for (int j = 0, seg = 0; j < P.m; ++j) {
    row_pass_r<true, MR>(P.radix[j], sm, ld, rows, L, span, x, D.twf + off, row_tw<MR>(D) + seg);
    seg += span;
    span /= P.radix[j];
    __syncthreads();
  }
  for (int i = threadIdx.x; i < rows * L; i += TH) {
    const int g = i / L, k = i - g * L;
    x[i] = sm[g * ld + sw(k)];
  }
}

// row_square_r16 with the pointwise square replaced by the product with the
// transformed rows F of another residue (row_forward_r16's output).
template <int TH, int MR>
__global__ void __launch_bounds__(TH) row_mul_r16(const TwoPassDesc* __restrict__ Ds, Passes P, int rows,
                                                  const uint64_t* __restrict__ F) {
  extern __shared__ __align__(16) uint64_t sm[];
  const TwoPassDesc& D = Ds[blockIdx.y];
  const int L = (int)D.n1, ld = padded(L);
  const size_t off = (size_t)blockIdx.x * rows * L;
  uint64_t* x = reinterpret_cast<uint64_t*>(D.x) + off;
  int span = L;
  for (int j = 0, seg = 0; j + 1 < P.m; ++j) {
    row_pass_r<true, MR>(P.radix[j], sm, ld, rows, L, span, x, D.twf + off, row_tw<MR>(D) + seg);
    seg += span;
    span /= P.radix[j];
    __syncthreads();
  }
  pass_r<3, MR>(P.radix[P.m - 1], sm, ld, rows, L, span, F + off);
  __syncthreads();
  for (int j = P.m - 2; j >= 0; --j) {
    span *= P.radix[j];
    row_pass_r<false, MR>(P.radix[j], sm, ld, rows, L, span, x, D.twi + off,
                      row_itw<MR>(D) + pass_table_offset(P, L, j));
    if (j) __syncthreads();
  }
}

// ------------------------------------------------------- rows of 5 L ----
//
// n = 5 * 2^k: a row holds n1 = 5 L words z[c'], c' = c + L j5.  Its transform
// (root omega_{5L} = omega_n^n2) splits as
//   Z[5 kL + k5] = sum_c omega_L^(c kL) omega_{5L}^(c k5) sum_j5 omega_5^(j5 k5) z[c + L j5]:
// a 5-point transform of the five words c, c + L, ..., c + 4L (fused with the
// 4-step twiddle as the row is loaded), a twiddle, and an L-point transform of
// each of the five planes (the passes above, bit-reversed output), whose last
// pass runs with the square as in row_square_r16.  The inverse runs the same
// steps backwards and stores the row; its factor 1/5 is in the unweights (1/n), and so is 1/64
// for the factors 4 of lazy::dft5.

// Mode 0: square (a squaring), 1: forward only (the operand F of a product,
// left in x in plane-major order), 2: product with F.  A CTA takes `rows`
// consecutive rows: plane k5 of row g at sm + (5 g + k5) ld.
template <int TH, int Mode>
__global__ void __launch_bounds__(TH) row5_r16(const TwoPassDesc* __restrict__ Ds, Passes P, int rows,
                                               const uint64_t* __restrict__ F) {
  extern __shared__ __align__(16) uint64_t sm[];
  const TwoPassDesc& D = Ds[blockIdx.y];
  const int L = (int)D.n1 / 5, ld = padded(L), W = 5 * L, lL = __ffs(L) - 1;
  const size_t off = (size_t)blockIdx.x * rows * W;
  uint64_t* x = reinterpret_cast<uint64_t*>(D.x) + off;
  const uint64_t* twf = D.twf + off;
  uint64_t c5[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) c5[k] = D.c5[k];
  // HBM -> planes: 4-step twiddle, 5-point transform, twiddle omega_5L^(c k5)
  for (int item = threadIdx.x; item < rows * L; item += TH) {
    const int g = item >> lL, c = item & (L - 1);
    const int i0 = g * W + c;
    lazy::W3 u[5];
    uint64_t v[5];
#pragma unroll
    for (int j5 = 0; j5 < 5; ++j5) u[j5] = lazy::mul3(x[i0 + j5 * L], twf[i0 + j5 * L]);
    lazy::dft5(u, c5, v);
    uint64_t* base = sm + 5 * g * ld + sw(c);
    base[0] = v[0];
#pragma unroll
    for (int k5 = 1; k5 < 5; ++k5) base[k5 * ld] = lazy::mul(v[k5], D.tw5[(k5 - 1) * L + c]);
  }
  __syncthreads();
  int span = L;
  const int last = Mode == 1 ? P.m : P.m - 1;
  for (int j = 0, seg = 0; j < last; ++j) {
    pass_r<0>(P.radix[j], sm, ld, 5 * rows, L, span, D.itw1 + seg);
    seg += span;
    span /= P.radix[j];
    __syncthreads();
  }
  if constexpr (Mode == 1) {
    for (int i = threadIdx.x; i < rows * W; i += TH) {
      const int p = i >> lL, e = i & (L - 1);
      x[i] = sm[p * ld + sw(e)];
    }
  } else {
    // last forward pass, square (or product with F) and first inverse pass
    if constexpr (Mode == 0)
      pass_r<2>(P.radix[P.m - 1], sm, ld, 5 * rows, L, span, nullptr);
    else
      pass_r<3>(P.radix[P.m - 1], sm, ld, 5 * rows, L, span, F + off);
    __syncthreads();
    for (int j = P.m - 2; j >= 0; --j) {
      span *= P.radix[j];
      pass_r<1>(P.radix[j], sm, ld, 5 * rows, L, span, D.iitw1 + pass_table_offset(P, L, j));
      __syncthreads();
    }
    // planes -> HBM: inverse twiddle, inverse 5-point transform, inverse 4-step twiddle
    const uint64_t* twi = D.twi + off;
    for (int item = threadIdx.x; item < rows * L; item += TH) {
      const int g = item >> lL, c = item & (L - 1);
      const int i0 = g * W + c;
      const uint64_t* base = sm + 5 * g * ld + sw(c);
      lazy::W3 u[5];
      uint64_t v[5];
      u[0] = lazy::from_word(base[0]);
#pragma unroll
      for (int k5 = 1; k5 < 5; ++k5) u[k5] = lazy::mul3(base[k5 * ld], D.itw5[(k5 - 1) * L + c]);
      lazy::dft5(u, c5, v);
      x[i0] = lazy::mul(v[0], twi[i0]);
      x[i0 + L] = lazy::mul(v[4], twi[i0 + L]);
      x[i0 + 2 * L] = lazy::mul(v[3], twi[i0 + 2 * L]);
      x[i0 + 3 * L] = lazy::mul(v[2], twi[i0 + 3 * L]);
      x[i0 + 4 * L] = lazy::mul(v[1], twi[i0 + 4 * L]);
    }
  }
}

// --------------------------------------------------------------- columns ----

// Threads per tile column.  A launch with CTAs enough to fill the GPU
// (throughput: a batch) gives each column one thread per radix-8 task of a pass
// (n2 / 8), at least a warp and at most 128, or 256 for columns of 4096 words
// (one 4-column CTA per SM): short columns then get small CTAs, many per SM,
// instead of CTAs whose threads mostly idle.  A launch with fewer CTAs than
// twice the SMs (one short test: latency) keeps 128 threads a column, whose
// row-wise steps (carries, weights, staging) then run in parallel.
// 16-point passes (columns of 1024 and more words) take half the threads at twice the registers.
template <int MR>
__host__ __device__ constexpr int col_tpc(uint32_t n2, bool latency) {
  if (MR == 16) return n2 >= 4096 ? 128 : 64;
  return n2 >= 4096 ? 256 : (n2 >= 1024 || latency ? 128 : (n2 == 512 ? 64 : 32));
}
inline bool col_latency_mode(const TwoPassDesc& d, uint32_t count) {
  return (uint64_t)d.ntiles * count < 2ull * device_sms();
}
// words of shared memory of a tile of T columns of L words (smem::Tile)
__host__ __device__ constexpr size_t tile_words(int L, int T) { return (size_t)T * (L + L / 8); }

// HBM -> shared memory without a register round trip: 16-byte cp.async of two adjacent columns of a
// row, so all of a thread's loads are in flight together.
template <int T>
__device__ __forceinline__ void tile_load(uint64_t* sm, const int64_t* x, int L, uint32_t n1, uint32_t c0) {
  for (int idx = threadIdx.x; idx < T / 2 * L; idx += blockDim.x) {
    const int r = idx / (T / 2), c = 2 * (idx % (T / 2));
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(sm + pos<Tile<T>>(r) + c);
    const int64_t* src = x + (size_t)r * n1 + c0 + c;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// HBM -> shared memory through L2 only (ld.global.cg): for a tile another CTA
// of the same launch has just written.
template <int T>
__device__ __forceinline__ void tile_load_cg(uint64_t* sm, const int64_t* x, int L, uint32_t n1, uint32_t c0) {
  for (int idx = threadIdx.x; idx < T * L; idx += blockDim.x) {
    const int r = idx / T, c = idx % T;
    sm[pos<Tile<T>>(r) + c] = (uint64_t)__ldcg(x + (size_t)r * n1 + c0 + c);
  }
}

// shared memory -> HBM, 16 bytes a thread
template <int T>
__device__ __forceinline__ void tile_store(const uint64_t* sm, int64_t* x, int L, uint32_t n1, uint32_t c0) {
#pragma unroll 4
  for (int idx = threadIdx.x; idx < T / 2 * L; idx += blockDim.x) {
    const int r = idx / (T / 2), c = 2 * (idx % (T / 2));
    *reinterpret_cast<ulonglong2*>(x + (size_t)r * n1 + c0 + c) =
        *reinterpret_cast<const ulonglong2*>(sm + pos<Tile<T>>(r) + c);
  }
}

// The separable weights (TwoPassDesc).  They replace weight, unweight and width tables of one
// entry per word (34 bytes a word and squaring of the column kernel's 66): the column factors ride
// in the 4-step twiddles, the row factors are a table of n2 entries that stays in the L1, and a
// word's own part is whether fa + fb wraps past n.
template <int T>
__device__ __forceinline__ void load_colf(const TwoPassDesc& D, uint32_t t0, uint32_t (&fa)[T]) {
  const uint4* src = reinterpret_cast<const uint4*>(D.colf + (size_t)t0 * T);
#pragma unroll
  for (int k = 0; k < T / 4; ++k) {
    const uint4 u = __ldg(src + k);
    fa[4 * k] = u.x;
    fa[4 * k + 1] = u.y;
    fa[4 * k + 2] = u.z;
    fa[4 * k + 3] = u.w;
  }
}

// A row of a tile, as 16-byte vectors.
template <int T>
__device__ __forceinline__ void load_row(const uint64_t* row, uint64_t (&v)[T]) {
  const ulonglong2* src = reinterpret_cast<const ulonglong2*>(row);
#pragma unroll
  for (int k = 0; k < T / 2; ++k) {
    const ulonglong2 u = src[k];
    v[2 * k] = u.x;
    v[2 * k + 1] = u.y;
  }
}
template <int T>
__device__ __forceinline__ void store_row(uint64_t* row, const uint64_t (&v)[T]) {
  ulonglong2* dst = reinterpret_cast<ulonglong2*>(row);
#pragma unroll
  for (int k = 0; k < T / 2; ++k) dst[k] = make_ulonglong2(v[2 * k], v[2 * k + 1]);
}

// f = fa + fb mod n; returns whether the sum wrapped
__device__ __forceinline__ bool weight_exponent(uint32_t fa, uint32_t fb, uint32_t n, uint32_t& f) {
  const uint32_t s = fa + fb;
  f = min(s, s - n);  // s - n wraps far above n while s < n
  return s >= n;
}

// ---- column tile bodies: tile t0 (T columns x L rows) staged in shared memory

// Carry-in from the run before each row's run, weight, forward column passes,
// store.  The tile's digits are in `sm`.  `cg_carries`: read the carries from L2
// (written by another CTA of the same launch).
template <int T, int MR>
__device__ __forceinline__ void forward_tile(const TwoPassDesc& D, const Passes& P, uint64_t* sm,
                                             uint32_t t0, bool apply_carries, bool cg_carries,
                                             uint32_t& status) {
  const int L = (int)D.n2;
  const uint32_t n = D.n, qmod = D.qmod, qdiv = D.qdiv;
  uint32_t fa[T];
  load_colf<T>(D, t0, fa);
  // per row: carry from the previous run, then weight (balanced digit -> field)
  for (int r = threadIdx.x; r < L; r += blockDim.x) {
    const size_t run = (size_t)t0 * L + r;
    const ulonglong2 wf = __ldg(D.rowf + 2 * r);
    uint64_t* row = sm + pos<Tile<T>>(r);
    uint64_t word[T];
    load_row<T>(row, word);
    int64_t carry = 0;
    if (apply_carries) {
      const int64_t* src = D.carry + (t0 > 0 ? run - L : (size_t)(D.ntiles - 1) * L + (r ? r - 1 : L - 1));
      carry = cg_carries ? __ldcg(src) : *src;
    }
#pragma unroll
    for (int c = 0; c < T; ++c) {
      uint64_t& v = word[c];
      int64_t d = (int64_t)v;
      uint32_t f;
      const bool wrapped = weight_exponent(fa[c], (uint32_t)wf.y, n, f);
      if (carry != 0) {
        if (c + 1 < T) {
          int64_t q;
          d = balance(d + carry, qdiv + (f < qmod), q);
          carry = q;
        } else {
          d += carry;
          if (carry > kAbsorbLimit || carry < -kAbsorbLimit) status |= kStatusCarryOverflow;
          carry = 0;
        }
      }
      // g^f = (g^fa / 2) g^fb 2^(not wrapped); digits stay below 2^31 (widths are at most 30)
      v = lazy::mul_digit(wrapped ? d : d + d, wf.x);
    }
    store_row<T>(row, word);
  }
  __syncthreads();
  int span = L;
  for (int j = 0, seg = 0; j < P.m; ++j) {
    pass_r<0, MR, Tile<T>>(P.radix[j], sm, 0, T, L, span, D.itw2 + seg);
    __syncthreads();
    seg += span;
    span /= P.radix[j];
  }
  tile_store<T>(sm, D.x, L, D.n1, t0 * T);
}

// Inverse column passes, unweight, carry each row's run of T words to balanced
// digits (minus two in the run of word 0), store the runs' outgoing carries.
// The tile's transform is in `sm`; its digits are left there.
template <int T, int MR>
__device__ __forceinline__ void inverse_tile(const TwoPassDesc& D, const Passes& P, uint64_t* sm,
                                             uint32_t t0, bool unsigned_mode) {
  const int L = (int)D.n2;
  int span = 1;
  for (int j = P.m - 1; j >= 0; --j) {
    span *= P.radix[j];
    pass_r<1, MR, Tile<T>>(P.radix[j], sm, 0, T, L, span, D.iitw2 + pass_table_offset(P, L, j));
    __syncthreads();
  }
  const uint32_t n = D.n, qmod = D.qmod, qdiv = D.qdiv;
  uint32_t fa[T];
  load_colf<T>(D, t0, fa);
  for (int r = threadIdx.x; r < L; r += blockDim.x) {
    const size_t run = (size_t)t0 * L + r;
    const uint32_t fb = (uint32_t)__ldg(D.rowf + 2 * r).y;
    const ulonglong2 u = __ldg(D.rowf + 2 * r + 1);
    uint64_t* row = sm + pos<Tile<T>>(r);
    uint64_t word[T];
    load_row<T>(row, word);
    int64_t carry = (!D.prp && t0 == 0 && r == 0) ? -2 : 0;
#pragma unroll
    for (int c = 0; c < T; ++c) {
      uint64_t& v = word[c];
      uint32_t f;
      const bool wrapped = weight_exponent(fa[c], fb, n, f);
      // g^-f / n = g^-fa (g^-fb / n) 2^(wrapped)
      uint64_t y = lazy::mul(v, wrapped ? u.y : u.x);
      if (unsigned_mode) y = gl::canon(y);
      v = (uint64_t)carry_digit(y, unsigned_mode, carry, qdiv + (f < qmod), carry);
    }
    store_row<T>(row, word);
    D.carry[run] = carry;
  }
  __syncthreads();
}

template <int T, int TH, int MR>
__global__ void __launch_bounds__(TH, min_blocks<TH, MR>()) col_forward_r16(
    const TwoPassDesc* __restrict__ Ds, Passes P, int apply_carries) {
  extern __shared__ __align__(16) uint64_t sm[];
  const TwoPassDesc& D = Ds[blockIdx.y];
  uint32_t status = 0;
  tile_load<T>(sm, D.x, (int)D.n2, D.n1, blockIdx.x * T);
  __syncthreads();
  forward_tile<T, MR>(D, P, sm, blockIdx.x, apply_carries != 0, false, status);
  if (status) atomicOr(D.status, status);
}

template <int T, int TH, int MR>
__global__ void __launch_bounds__(TH, min_blocks<TH, MR>()) col_inverse_r16(
    const TwoPassDesc* __restrict__ Ds, Passes P, int unsigned_mode) {
  extern __shared__ __align__(16) uint64_t sm[];
  const TwoPassDesc& D = Ds[blockIdx.y];
  tile_load<T>(sm, D.x, (int)D.n2, D.n1, blockIdx.x * T);
  __syncthreads();
  inverse_tile<T, MR>(D, P, sm, blockIdx.x, unsigned_mode != 0);
  tile_store<T>(sm, D.x, (int)D.n2, D.n1, blockIdx.x * T);
}

// ---- carry-fused column kernel: col_inverse of one squaring and col_forward
// of the next in one launch, the tile staying in shared memory in between.
//
// A tile's second half needs the carries of the tile before it (the runs of
// the same rows); tile 0 needs those of the LAST tile (the runs of the rows
// before).  CTAs take tickets in start order (an atomic counter) and no CTA
// ever waits for a CTA that took a later ticket, so every wait ends whatever
// else holds the GPU's CTA slots (other tests, other launches):
//   ticket 0:          first half of the last tile (its digits go back to x,
//                      flag), first half of tile 0 (flag), then tile 0's
//                      second half with the last tile's carries it has just
//                      made itself;
//   ticket t, 0<t<T-1: first half of tile t (flag), wait for tile t-1's flag,
//                      second half;
//   ticket T-1:        wait for the last tile's flag (ticket 0 has stored its
//                      digits) and tile T-2's flag, reload the digits, second
//                      half.
// Flags hold a per-launch epoch, so nothing is cleared between launches.  Every
// wait is bounded in time and reported.
//
// fuse[0]: ticket counter, fuse[1]: epoch, fuse[2 + t]: flag of tile t.
constexpr uint64_t kWaitLimitNs = 2000000000ull;  // 2 s: far above any launch; then report, never hang

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void publish_flag(uint32_t* flag, uint32_t v) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(flag), "r"(v) : "memory");
  }
}

// Thread 0 polls the flag (acquire), the CTA waits at the barrier.  Gives up
// after kWaitLimitNs, or at once when another CTA already gave up.
__device__ __forceinline__ void wait_flag(const uint32_t* flag, uint32_t want, uint32_t* status) {
  if (threadIdx.x == 0) {
    const uint64_t start = global_ns();
    uint32_t v = 0, iters = 0;
    while (true) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
      if (v == want) break;
      if ((++iters & 63) == 0) {
        if (*(volatile uint32_t*)status & kStatusFuseTimeout) break;
        if (global_ns() - start > kWaitLimitNs) {
          atomicOr(status, kStatusFuseTimeout);
          break;
        }
      }
      __nanosleep(100);
    }
  }
  __syncthreads();
}

template <int T, int TH, int MR, bool Dense>
__global__ void __launch_bounds__(TH, min_blocks<TH, MR, Dense>()) col_fused_r16(
    const TwoPassDesc* __restrict__ Ds, Passes P) {
  extern __shared__ __align__(16) uint64_t sm[];
  __shared__ uint32_t s_ticket, s_epoch;
  const TwoPassDesc& D = Ds[blockIdx.y];
  const int L = (int)D.n2;
  const uint32_t n1 = D.n1, ntiles = D.ntiles, last = ntiles - 1;
  uint32_t* ctl = D.fuse;
  if (threadIdx.x == 0) {
    // the epoch is read before the ticket: the last ticket's CTA advances it
    // only after every CTA of the launch has taken its ticket
    uint32_t e;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(e) : "l"(ctl + 1) : "memory");
    s_epoch = e;
    s_ticket = atomicAdd(ctl, 1u);
  }
  __syncthreads();
  const uint32_t ticket = s_ticket, ready = s_epoch + 1;
  if (ticket >= ntiles || ntiles < 2) {  // a counter left over from a launch that did not finish: report, touch nothing
    if (threadIdx.x == 0) atomicOr(D.status, kStatusFuseTimeout);
    return;
  }
  uint32_t status = 0;
  const bool is_last = ticket == last;

  // first halves, each inverse_tile / forward_tile body instantiated once (the
  // kernel stays small for the instruction cache): ticket 0 does the last
  // tile's and then tile 0's, ticket t < T-1 its own, ticket T-1 none
  const int ninv = is_last ? 0 : (ticket == 0 ? 2 : 1);
  for (int i = 0; i < ninv; ++i) {
    const bool lasttile = ticket == 0 && i == 0;
    const uint32_t tile = lasttile ? last : ticket;
    tile_load<T>(sm, D.x, L, n1, tile * T);
    __syncthreads();
    inverse_tile<T, MR>(D, P, sm, tile, false);
    // the last tile's digits wait in x for the last ticket
    if (lasttile) tile_store<T>(sm, D.x, L, n1, last * T);
    publish_flag(ctl + 2 + tile, ready);
  }
  if (is_last) {
    // the last tile's first half was done by ticket 0 (digits in x)
    wait_flag(ctl + 2 + last, ready, D.status);
    tile_load_cg<T>(sm, D.x, L, n1, last * T);
  }
  // second half: carries in from the tile before (tile 0: the last tile, made
  // by this CTA), weight, forward column transform
  if (ticket > 0) wait_flag(ctl + 2 + ticket - 1, ready, D.status);
  forward_tile<T, MR>(D, P, sm, ticket, true, true, status);
  if (is_last && threadIdx.x == 0) {
    // every ticket of this launch is taken and every CTA has read the epoch
    ctl[0] = 0;
    __threadfence();
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(ctl + 1), "r"(ready) : "memory");
  }
  if (status) atomicOr(D.status, status);
}

// Raise a kernel's dynamic shared-memory cap once per device (the cap does not
// change occupancy; the launch's own size does), so launches made while a
// stream is being captured into a graph issue no attribute calls.
template <typename K>
cudaError_t ensure_smem(K* kernel, size_t smem) {
  static std::mutex mu;
  static std::map<std::pair<const void*, int>, size_t> done;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(mu);
  const auto key = std::make_pair((const void*)kernel, dev);
  auto it = done.find(key);
  if (it != done.end() && it->second >= smem) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) done[key] = smem;
  return e;
}

// Rows per row-kernel CTA: up to 4096 words of rows (the CTA's 256 threads
// then have two tasks each per pass), fewer while the launch would have fewer
// CTAs than the GPU has SMs (one test: latency) or than four per SM (a batch
// of `count` tests: throughput).
int row_rows_per_cta(int L, int n2, uint32_t count) {
  int rows = 4096 / L;
  if (rows < 1) rows = 1;
  const int sms = (int)device_sms();
  const long want = count > 1 ? 4L * sms : sms;
  while (rows > 1 && (long)(n2 / rows) * (long)count < want) rows /= 2;
  return rows;
}

}  // namespace

std::vector<uint32_t> r16_pass_radices(uint32_t log2L, uint32_t radix) {
  const Passes p = make_passes((int)log2L, radix == 16 ? 4 : 3);
  std::vector<uint32_t> r;
  for (int j = 0; j < p.m; ++j) r.push_back((uint32_t)p.radix[j]);
  return r;
}

// Rows up to 2^14 words (139 KB of shared memory, one CTA per SM) and columns
// up to 2^12 (four columns: 139 KB): with B200's 227 KB per CTA the 2^25 and
// 2^26 lengths stay two-pass, where the reference needs 3-factor plans
// (ntt_lengths.cu:118-127).
bool r16_supported(uint32_t log2n1, uint32_t log2n2) {
  return log2n2 >= 6 && log2n2 <= 12 && log2n1 >= 7 && log2n1 <= 14 && log2n1 >= log2n2;
}

uint32_t r16_tile(uint32_t log2n2) { return log2n2 >= 12 ? 4 : 8; }

// Words a carry run needs: the outgoing carry of a run is below 2^(log2 n + W)
// in magnitude (W = ceil(q / n)), each word it ripples through takes off at
// least w_min - 1 bits, and the last word absorbs the remaining +-1.
uint32_t r16_run_words_needed(uint32_t exponent, uint32_t n) {
  uint32_t log2n = 0;
  while ((1ull << log2n) < n) ++log2n;
  const uint32_t wmax = (exponent + n - 1) / n, wmin = exponent / n;
  if (wmin < 3) return 64;
  return (log2n + wmax + wmin - 2) / (wmin - 1) + 1;
}

// Passes of 16 points save one pass (and a quarter of the general products) of a transform of 1024,
// 2048 or 4096 words, at twice the registers.  Columns gain from it (col_fused, us, 8 -> 16 points:
// n2 = 1024 40.8 -> 36.9 at n = 2^20, 2048 188.8 -> 178 at 2^23, 4096 408 -> 389 at 2^24 and 1603 ->
// 1509 at 2^26; 512 words save no pass: 24.5 -> 28.5 at 2^19).  Lengths 5 * 2^k have no radix option;
// their columns follow the same line.
uint32_t r16_col_radix(uint32_t plan_radix, bool five, uint32_t n2) {
  return (plan_radix == 16 || five) && n2 >= 1024 ? 16 : 8;
}
// Rows of 1024 and 2048 words gain only in a launch that leaves registers idle, below four CTAs an SM
// (row_square, us: 32.7 -> 26.5 at 2^20, 51.1 -> 47.0 at 2^21; 1024 CTAs of 2048 words, 2^22, 88 -> 104);
// such plans keep the pass tables of both radices.  Rows of 4096 words and more lose (157.9 -> 182.1 at
// 2^23): their first and last passes, whose 16 words and 16 twiddles a task come from HBM, find too few
// warps to hide it.
uint32_t r16_row_radix(uint32_t plan_radix, uint32_t n1) {
  return plan_radix == 16 && (n1 == 1024 || n1 == 2048) ? 16 : 8;
}
bool rows16(const TwoPassDesc& d, uint32_t count) {
  return r16_row_radix(d.radix, d.n1) == 16 &&
         (uint64_t)(d.n2 / row_rows_per_cta((int)d.n1, (int)d.n2, count)) * count < 4ull * device_sms();
}
bool cols16(const TwoPassDesc& d) { return r16_col_radix(d.radix, d.five != 0, d.n2) == 16; }

template <int TH, int MR>
cudaError_t row_square_t(const TwoPassDesc& d, const TwoPassDesc* dd, uint32_t count, cudaStream_t s) {
  const int L = (int)d.n1, rows = row_rows_per_cta(L, (int)d.n2, count);
  const size_t smem = (size_t)rows * padded(L) * 8;
  cudaError_t e = ensure_smem(row_square_r16<TH, MR>, smem);
  if (e != cudaSuccess) return e;
  row_square_r16<TH, MR><<<dim3(d.n2 / rows, count), TH, smem, s>>>(dd, make_passes((int)d.log2n1, MR == 16 ? 4 : 3), rows);
  return cudaGetLastError();
}

template <int TH, int MR>
cudaError_t row_forward_t(const TwoPassDesc& d, const TwoPassDesc* dd, cudaStream_t s) {
  const int L = (int)d.n1, rows = row_rows_per_cta(L, (int)d.n2, 1);
  const size_t smem = (size_t)rows * padded(L) * 8;
  cudaError_t e = ensure_smem(row_forward_r16<TH, MR>, smem);
  if (e != cudaSuccess) return e;
  row_forward_r16<TH, MR><<<dim3(d.n2 / rows, 1), TH, smem, s>>>(dd, make_passes((int)d.log2n1, MR == 16 ? 4 : 3), rows);
  return cudaGetLastError();
}

template <int TH, int MR>
cudaError_t row_mul_t(const TwoPassDesc& d, const TwoPassDesc* dd, const uint64_t* F, cudaStream_t s) {
  const int L = (int)d.n1, rows = row_rows_per_cta(L, (int)d.n2, 1);
  const size_t smem = (size_t)rows * padded(L) * 8;
  cudaError_t e = ensure_smem(row_mul_r16<TH, MR>, smem);
  if (e != cudaSuccess) return e;
  row_mul_r16<TH, MR><<<dim3(d.n2 / rows, 1), TH, smem, s>>>(dd, make_passes((int)d.log2n1, MR == 16 ? 4 : 3), rows, F);
  return cudaGetLastError();
}

// 16-point passes: rows of 1024 or 2048 words only (r16_row_radix), 256 threads and fewer
template <int MR>
cudaError_t row_forward_m(const TwoPassDesc& d, const TwoPassDesc* dd, cudaStream_t s) {
  if constexpr (MR == 16) return row_forward_t<256, MR>(d, dd, s);
  else switch (row_threads_for((int)d.n1)) {
    case 256: return row_forward_t<256, MR>(d, dd, s);
    case 512: return row_forward_t<512, MR>(d, dd, s);
    default: return row_forward_t<1024, MR>(d, dd, s);
  }
}

template <int MR>
cudaError_t row_mul_m(const TwoPassDesc& d, const TwoPassDesc* dd, const uint64_t* F, cudaStream_t s) {
  if constexpr (MR == 16) return row_mul_t<256, MR>(d, dd, F, s);
  else switch (row_threads_for((int)d.n1)) {
    case 256: return row_mul_t<256, MR>(d, dd, F, s);
    case 512: return row_mul_t<512, MR>(d, dd, F, s);
    default: return row_mul_t<1024, MR>(d, dd, F, s);
  }
}

template <int MR>
cudaError_t row_square_m(const TwoPassDesc& d, const TwoPassDesc* dd, uint32_t count, cudaStream_t s) {
  const int rows = row_rows_per_cta((int)d.n1, (int)d.n2, count);
  const bool latency = (uint64_t)(d.n2 / rows) * count < 2ull * device_sms();
  switch (row_square_threads((int)d.n1, rows, latency)) {
    case 64: return row_square_t<64, MR>(d, dd, count, s);
    case 128: return row_square_t<128, MR>(d, dd, count, s);
    case 256: return row_square_t<256, MR>(d, dd, count, s);
    default: break;
  }
  if constexpr (MR == 8) {
    switch (row_square_threads((int)d.n1, rows, latency)) {
      case 32: return row_square_t<32, MR>(d, dd, count, s);
      case 512: return row_square_t<512, MR>(d, dd, count, s);
      default: return row_square_t<1024, MR>(d, dd, count, s);
    }
  }
  return cudaErrorInvalidConfiguration;
}

// Rows of 5 L words (radix-8 passes) per CTA: as many as fit 4096 words (a
// power of two), fewer while the launch would have fewer CTAs than the SMs (one
// test) or than four per SM (a batch of `count`); 128 threads for up to 1280
// words a CTA, 256 up to 5120, then 512 and 1024.
template <int Mode>
cudaError_t row5_launch(const TwoPassDesc& d, const TwoPassDesc* dd, uint32_t count,
                        const uint64_t* F, cudaStream_t s) {
  const int L = (int)d.n1 / 5;
  int rows = 1;
  while (rows * 2 * (int)d.n1 <= 4096 && rows * 2 <= (int)d.n2) rows *= 2;
  const long want = count > 1 ? 4L * device_sms() : (long)device_sms();
  while (rows > 1 && (long)(d.n2 / rows) * (long)count < want) rows /= 2;
  const size_t smem = (size_t)5 * rows * padded(L) * 8;
  const Passes P = make_passes((int)d.log2n1, 3);
  const dim3 grid(d.n2 / rows, count);
  const int words = rows * (int)d.n1;
  auto go = [&](auto kernel, int th) {
    cudaError_t e = ensure_smem(kernel, smem);
    if (e != cudaSuccess) return e;
    kernel<<<grid, th, smem, s>>>(dd, P, rows, F);
    return cudaGetLastError();
  };
  if (words <= 1280) return go(row5_r16<128, Mode>, 128);
  if (words <= 5120) return go(row5_r16<256, Mode>, 256);
  if (words <= 10240) return go(row5_r16<512, Mode>, 512);
  return go(row5_r16<1024, Mode>, 1024);
}

cudaError_t launch_row_forward_r16(const TwoPassDesc& d, const TwoPassDesc* dd, cudaStream_t s) {
  if (d.five) return row5_launch<1>(d, dd, 1, nullptr, s);
  return rows16(d, 1) ? row_forward_m<16>(d, dd, s) : row_forward_m<8>(d, dd, s);
}

cudaError_t launch_row_mul_r16(const TwoPassDesc& d, const TwoPassDesc* dd, const uint64_t* F,
                               cudaStream_t s) {
  if (d.five) return row5_launch<2>(d, dd, 1, F, s);
  return rows16(d, 1) ? row_mul_m<16>(d, dd, F, s) : row_mul_m<8>(d, dd, F, s);
}

cudaError_t launch_row_square_r16(const TwoPassDesc& d, const TwoPassDesc* dd, uint32_t count,
                                  cudaStream_t s) {
  if (d.five) return row5_launch<0>(d, dd, count, nullptr, s);
  return rows16(d, count) ? row_square_m<16>(d, dd, count, s) : row_square_m<8>(d, dd, count, s);
}

// The column kernels' thread count for a tile of T columns of n2 words.
template <int T, int MR, class F>
cudaError_t col_dispatch(uint32_t n2, bool latency, F&& f) {
  switch (T * col_tpc<MR>(n2, latency)) {
    case 128:
      if constexpr (T == 4 && MR == 8) return f(std::integral_constant<int, 128>{});
      break;
    case 256:
      if constexpr (T == 4 || MR == 8) return f(std::integral_constant<int, 256>{});
      break;
    case 512: return f(std::integral_constant<int, 512>{});
    case 1024:
      if constexpr (MR == 8) return f(std::integral_constant<int, 1024>{});
      break;
    default: break;
  }
  return cudaErrorInvalidConfiguration;
}
template <int T, int TH, int MR>
cudaError_t col_forward_t(const TwoPassDesc& d, const TwoPassDesc* dd, uint32_t count, bool apply,
                          cudaStream_t s) {
  const size_t smem = tile_words((int)d.n2, T) * 8;
  cudaError_t e = ensure_smem(col_forward_r16<T, TH, MR>, smem);
  if (e != cudaSuccess) return e;
  col_forward_r16<T, TH, MR><<<dim3(d.ntiles, count), TH, smem, s>>>(dd, make_passes((int)d.log2n2, MR == 16 ? 4 : 3), apply ? 1 : 0);
  return cudaGetLastError();
}

template <int T, int TH, int MR>
cudaError_t col_inverse_t(const TwoPassDesc& d, const TwoPassDesc* dd, uint32_t count,
                          bool unsigned_mode, cudaStream_t s) {
  const size_t smem = tile_words((int)d.n2, T) * 8;
  cudaError_t e = ensure_smem(col_inverse_r16<T, TH, MR>, smem);
  if (e != cudaSuccess) return e;
  col_inverse_r16<T, TH, MR><<<dim3(d.ntiles, count), TH, smem, s>>>(dd, make_passes((int)d.log2n2, MR == 16 ? 4 : 3), unsigned_mode ? 1 : 0);
  return cudaGetLastError();
}

template <int T, int TH, int MR, bool Dense>
cudaError_t col_fused_t(const TwoPassDesc& d, const TwoPassDesc* dd, uint32_t count, cudaStream_t s) {
  const size_t smem = tile_words((int)d.n2, T) * 8;
  cudaError_t e = ensure_smem(col_fused_r16<T, TH, MR, Dense>, smem);
  if (e != cudaSuccess) return e;
  col_fused_r16<T, TH, MR, Dense><<<dim3(d.ntiles, count), TH, smem, s>>>(dd, make_passes((int)d.log2n2, MR == 16 ? 4 : 3));
  return cudaGetLastError();
}

// 16-point passes of 4-word tiles up to 2048 rows (73 KB: three fit an SM): three CTAs an SM instead
// of two where the launch has eight tiles an SM and more.  col_fused, two -> three, us: 2560 tiles of 1024
// rows (n = 5 * 2^21) 246.7 -> 223.2; 512 of 2048 (2^22) 108.0 -> 113.3, 512 of 1024 (2^21) 59.2 -> 65.8, where
// the third CTA saves no wave.  The line keeps clear of those: 1024 tiles of 2048 (one test at 2^23) lie below it
// and take two, although three would be 180.9 -> 177.6 there; other launches of 600 to 1184 tiles
// (several tests) have not been measured.
bool col_dense(const TwoPassDesc& d, uint32_t count) {
  return d.tile == 4 && d.n2 <= 2048 && (uint64_t)d.ntiles * count >= 8ull * device_sms();
}

// Tests per launch (the grid's y extent).  A CTA of the fused kernel waits only
// for CTAs that started before it, so the count is not bounded by how many
// CTAs the GPU holds at once.
constexpr uint32_t kFusedTestsPerLaunch = 1024;

template <int T, int MR>
cudaError_t col_fused_tm(const TwoPassDesc& d, const TwoPassDesc* dd, uint32_t count, cudaStream_t s) {
  return col_dispatch<T, MR>(d.n2, col_latency_mode(d, count), [&](auto th) {
    constexpr int TH = decltype(th)::value;
    if constexpr (MR == 16 && T == 4 && TH == 256)
      if (col_dense(d, count)) return col_fused_t<T, TH, MR, true>(d, dd, count, s);
    return col_fused_t<T, TH, MR, false>(d, dd, count, s);
  });
}

template <int MR>
cudaError_t col_fused_m(const TwoPassDesc& d, const TwoPassDesc* dd, uint32_t count, cudaStream_t s) {
  for (uint32_t first = 0; first < count; first += kFusedTestsPerLaunch) {
    const uint32_t c = count - first < kFusedTestsPerLaunch ? count - first : kFusedTestsPerLaunch;
    const cudaError_t e = d.tile == 8 ? col_fused_tm<8, MR>(d, dd + first, c, s)
                                      : col_fused_tm<4, MR>(d, dd + first, c, s);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

template <int MR>
cudaError_t col_forward_m(const TwoPassDesc& d, const TwoPassDesc* dd, uint32_t count, bool apply,
                          cudaStream_t s) {
  const bool latency = col_latency_mode(d, count);
  if (d.tile == 8)
    return col_dispatch<8, MR>(d.n2, latency,
                           [&](auto th) { return col_forward_t<8, decltype(th)::value, MR>(d, dd, count, apply, s); });
  return col_dispatch<4, MR>(d.n2, latency,
                         [&](auto th) { return col_forward_t<4, decltype(th)::value, MR>(d, dd, count, apply, s); });
}

template <int MR>
cudaError_t col_inverse_m(const TwoPassDesc& d, const TwoPassDesc* dd, uint32_t count,
                          bool unsigned_mode, cudaStream_t s) {
  const bool latency = col_latency_mode(d, count);
  if (d.tile == 8)
    return col_dispatch<8, MR>(d.n2, latency, [&](auto th) {
      return col_inverse_t<8, decltype(th)::value, MR>(d, dd, count, unsigned_mode, s);
    });
  return col_dispatch<4, MR>(d.n2, latency, [&](auto th) {
    return col_inverse_t<4, decltype(th)::value, MR>(d, dd, count, unsigned_mode, s);
  });
}

cudaError_t launch_col_fused_r16(const TwoPassDesc& d, const TwoPassDesc* dd, uint32_t count,
                                 cudaStream_t s) {
  return cols16(d) ? col_fused_m<16>(d, dd, count, s) : col_fused_m<8>(d, dd, count, s);
}

cudaError_t launch_col_forward_r16(const TwoPassDesc& d, const TwoPassDesc* dd, uint32_t count,
                                   bool apply, cudaStream_t s) {
  return cols16(d) ? col_forward_m<16>(d, dd, count, apply, s)
                       : col_forward_m<8>(d, dd, count, apply, s);
}

cudaError_t launch_col_inverse_r16(const TwoPassDesc& d, const TwoPassDesc* dd, uint32_t count,
                                   bool unsigned_mode, cudaStream_t s) {
  return cols16(d) ? col_inverse_m<16>(d, dd, count, unsigned_mode, s)
                       : col_inverse_m<8>(d, dd, count, unsigned_mode, s);
}

}  // namespace lnt
