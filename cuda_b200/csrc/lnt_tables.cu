// Precomputed tables: IBDWT weights/unweights and 4-step twiddles.
//
// Replaces common/pre_calculation.cu:23-36 (calc_weights_widths) and :69-77
// (calc_brev_factors).  The weights are the same field elements as the
// reference's: w_j = 7^(((p-1)/192/n) * 5 * (n - r_j)), r_j = q j mod n, w_0 = 1,
// uw_j = (w_j n)^-1, uw_0 = n^-1.  With g = 7^(((p-1)/192/n) * 5) (g^n = 2),
// uw_j = g^r_j / (2n) for j > 0.  The weight of word j thus places it at bit
// ceil(qj/n) when r_j != 0; words with r_j = 0, j > 0 (q sharing a factor with
// n) sit exactly on bit qj/n and take weight 1.  The widths (lnt_policy.cpp,
// word_widths) are the exact integer differences of those bits, so every word
// starts where its weight says.
#include "lnt_internal.h"
#include "goldilocks.cuh"
#include "lazy_core.cuh"

namespace lnt {

namespace {

__global__ void weights_kernel(uint32_t exponent, uint32_t n, uint64_t g, uint64_t inv_n,
                               uint64_t inv_2n, uint64_t* w, uint64_t* uw) {
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  if (j == 0) {
    w[0] = 1;
    uw[0] = inv_n;
    return;
  }
  const uint32_t r = (uint32_t)(((uint64_t)exponent * j) % n);
  if (r == 0) {
    // qj/n is a whole bit: the word starts exactly there (weight 1).  The formula
    // below would give g^n = 2, one bit off; this happens for j > 0 only when q
    // shares a factor with n (an even q, or q divisible by 5 at n = 5 * 2^k).
    w[j] = 1;
    uw[j] = inv_n;
    return;
  }
  w[j] = gl::pow(g, (uint64_t)(n - r));
  uw[j] = gl::mul(gl::pow(g, (uint64_t)r), inv_2n);
}

// twf[row * n1 + j1] = omega_n^(j1 * k2) with k2 = bit-reverse(row) over log2n2
// bits: the frequency that the forward column NTT leaves in memory row `row`.
__global__ void twiddle_kernel(uint32_t n1, uint32_t n2, uint32_t log2n2, uint64_t root,
                               uint64_t iroot, const ulonglong2* colw, uint64_t* twf, uint64_t* twi) {
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (size_t)n1 * n2) return;
  const uint32_t row = (uint32_t)(idx / n1), j1 = (uint32_t)(idx % n1);
  const uint32_t k2 = __brev(row) >> (32 - log2n2);
  const uint64_t e = (uint64_t)j1 * k2;
  uint64_t f = gl::pow(root, e), i = gl::pow(iroot, e);
  if (colw) {
    f = gl::mul(f, colw[j1].x);
    i = gl::mul(i, colw[j1].y);
  }
  twf[idx] = f;
  twi[idx] = i;
}

// f(m) = -q m mod n for the columns (m = j1 < n1) and the rows (m = n1 j2)
__global__ void weight_factor_kernel(uint32_t exponent, uint32_t n1, uint32_t n2, uint64_t g, uint64_t ginv,
                                     uint64_t inv2, uint64_t inv_n, ulonglong2* rowf, uint32_t* colf,
                                     ulonglong2* colw) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, n = n1 * n2;
  auto neg_mod = [&](uint64_t m) {
    const uint32_t r = (uint32_t)((uint64_t)exponent * m % n);
    return r ? n - r : 0u;
  };
  if (i < n1) {
    const uint32_t f = neg_mod(i);
    colf[i] = f;
    colw[i] = make_ulonglong2(gl::mul(gl::pow(g, f), inv2), gl::pow(ginv, f));
  }
  if (i < n2) {
    const uint32_t f = neg_mod((uint64_t)n1 * i);
    const uint64_t u = gl::mul(gl::pow(ginv, f), inv_n);
    rowf[2 * i] = make_ulonglong2(gl::pow(g, f), f);
    rowf[2 * i + 1] = make_ulonglong2(u, gl::add(u, u));
  }
}

}  // namespace

cudaError_t launch_weight_factors(uint32_t exponent, uint32_t n1, uint32_t n2, ulonglong2* rowf, uint32_t* colf,
                                  ulonglong2* colw, cudaStream_t s) {
  const uint32_t n = n1 * n2, m = n1 > n2 ? n1 : n2;
  const uint64_t g = gl::pow(7, ((gl::P - 1) / 192 / n) * 5ull);  // g^n = 2
  const uint64_t scale = n % 5 ? n : n * lazy::kDft5Scale;
  weight_factor_kernel<<<(m + 127) / 128, 128, 0, s>>>(exponent, n1, n2, g, gl::inv(g), gl::inv(2), gl::inv(scale),
                                                       rowf, colf, colw);
  return cudaGetLastError();
}

namespace {
__global__ void power_kernel(uint32_t n, uint64_t root, uint64_t* pw) {
  const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < n) pw[e] = gl::pow(root, e);
}
}  // namespace

cudaError_t launch_powers(uint32_t n, uint64_t* pw, cudaStream_t s) {
  power_kernel<<<(n + 127) / 128, 128, 0, s>>>(n, gl::pow(554, (gl::P - 1) / n), pw);
  return cudaGetLastError();
}

cudaError_t launch_weights(uint32_t exponent, uint32_t n, uint64_t* w, uint64_t* uw,
                           cudaStream_t s) {
  const uint64_t c = ((gl::P - 1) / 192 / n) * 5ull;
  const uint64_t g = gl::pow(7, c);
  const uint64_t inv_n = gl::inv(n), inv_2n = gl::inv(2ull * n);
  const uint32_t threads = 256, blocks = (n + threads - 1) / threads;
  weights_kernel<<<blocks, threads, 0, s>>>(exponent, n, g, inv_n, inv_2n, w, uw);
  return cudaGetLastError();
}

namespace {
// tw5[(k5 - 1) L + c] = omega_{5L}^(k5 c): the twiddle between the 5-point
// transform of the words c + L j5 and the L-point transform of plane k5
__global__ void five_twiddle_kernel(uint32_t L, uint64_t root, uint64_t iroot, uint64_t* tw5,
                                    uint64_t* itw5) {
  const uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= 4 * L) return;
  const uint64_t e = (uint64_t)(idx / L + 1) * (idx % L);
  tw5[idx] = gl::pow(root, e);
  itw5[idx] = gl::pow(iroot, e);
}
}  // namespace

cudaError_t launch_five_twiddles(uint32_t L, uint64_t* tw5, uint64_t* itw5, uint64_t c5[4],
                                 cudaStream_t s) {
  // omega_{5L} = 554^((p-1)/5L) = omega_n^n2, the same root family as every other table
  const uint64_t root = gl::pow(554, (gl::P - 1) / (5ull * L)), iroot = gl::inv(root);
  lazy::dft5_constants(gl::pow(root, L), c5);
  five_twiddle_kernel<<<(4 * L + 255) / 256, 256, 0, s>>>(L, root, iroot, tw5, itw5);
  return cudaGetLastError();
}

cudaError_t launch_twiddles(uint32_t n1, uint32_t n2, uint32_t log2n2, const ulonglong2* colw, uint64_t* twf,
                            uint64_t* twi, cudaStream_t s) {
  const uint64_t n = (uint64_t)n1 * n2;
  const uint64_t root = gl::pow(554, (gl::P - 1) / n);
  const uint64_t iroot = gl::inv(root);
  const uint32_t threads = 256;
  const uint64_t blocks = (n + threads - 1) / threads;
  twiddle_kernel<<<(unsigned)blocks, threads, 0, s>>>(n1, n2, log2n2, root, iroot, colw, twf, twi);
  return cudaGetLastError();
}

}  // namespace lnt
