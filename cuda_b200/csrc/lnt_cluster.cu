// Cluster-resident squaring loop: one residue of 512 ... 32768 words over the shared memories
// of a thread-block cluster, for every squaring of a launch.
//
// One test alone on one SM (lnt_resident.cu) leaves 147 SMs idle and is bound by the latency of
// its passes, not by their work (n = 2048: 9.0 us a squaring, about 3 us of issue slots); a small
// two-pass plan (lnt_radix16.cu) pays three dependent launches a squaring (n = 8192: 15.4 us).
// Here C CTAs of a cluster hold n / C = m words each:
//   natural layout: CTA c keeps the words k m + c m / C + u, k < C, u < m / C (C segments);
//   block layout:   CTA r keeps the r-th block of m words after a first pass of radix C.
// A squaring is: carry-in and weight, radix-C pass (writes go to the CTAs that own the blocks,
// through distributed shared memory), the passes of a length-m transform, square, inverse passes
// (the last one writes to the natural owners), inverse radix-C pass, unweight and carry runs: three
// exchanges and about eight CTA barriers, no global memory access.  (With cluster barriers in place
// of the counted stores of `send`: 5.45 us against 5.09 at n = 2048.)  Twiddles, weights and
// unweights sit in shared memory (69 bytes a word with the two buffers: up to m = 2048).
//
// Replaces the reference's FFT_1SMEM pool as lnt_resident.cu does (kernel_pool.cu:31-38).
#include <algorithm>
#include <mutex>
#include <map>

#include "carry.cuh"
#include "cluster_exchange.h"
#include "lazy_core.cuh"
#include "lnt_internal.h"
#include "smem_passes.cuh"

namespace lnt {

namespace {

using namespace smem;

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// An exchange between the CTAs of a cluster: every word is stored asynchronously into the receiving
// CTA's shared memory and counts there towards an mbarrier, so a CTA goes on when its own words have
// arrived (one crossing), not when the whole cluster has stored, fenced and met in a barrier.  No
// buffer needs a second barrier before it is written again: a CTA sends only what follows from data
// of every CTA that still had to read the place.
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t remote_addr(uint32_t a, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void send(const void* local, const uint64_t* bar, uint32_t rank, uint64_t v) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.u64 [%0], %1, [%2];" ::"r"(
                   remote_addr(smem_addr(local), rank)),
               "l"(v), "r"(remote_addr(smem_addr(bar), rank))
               : "memory");
}
__device__ __forceinline__ void expect_bytes(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
// takes bytes that will not be sent off the barrier's count
__device__ __forceinline__ void complete_bytes(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.complete_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void store_remote(const void* local, uint32_t rank, uint64_t v) {
  asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(remote_addr(smem_addr(local), rank)), "l"(v) : "memory");
}
// Every thread of the CTA waits for the barrier's phase, at most wait_ns (kClusterWaitNs, two seconds:
// an exchange takes under a microsecond).  A wait that gives up raises kStatusClusterTimeout, and at its
// next barrier the whole CTA leaves the loop (gave_up); the CTAs that then miss its words give up in turn.
__device__ __forceinline__ void await_phase(uint64_t* bar, uint32_t parity, const uint64_t& wait_ns, uint32_t& status) {
  uint64_t start = 0;
  for (uint32_t i = 1; !(status & kStatusClusterTimeout); ++i) {
    uint32_t done;
    asm volatile("{\n\t"
                 ".reg .pred p;\n\t"
                 "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t"
                 "}"
                 : "=r"(done)
                 : "r"(smem_addr(bar)), "r"(parity)
                 : "memory");
    if (done) return;
    if ((i & 15) == 0) {
      uint64_t now;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
      if (!start) start = now;
      if (now - start > wait_ns) status |= kStatusClusterTimeout;
    }
  }
}
// a barrier of the CTA that also tells whether a wait of any of its threads gave up
__device__ __forceinline__ bool gave_up(uint32_t status) { return __syncthreads_or((int)(status & kStatusClusterTimeout)) != 0; }

__device__ __forceinline__ int brev_bits(int i, int bits) { return bits ? (int)(__brev((unsigned)i) >> (32 - bits)) : 0; }

// Everything a CTA keeps, in words of shared memory.
struct Layout {
  uint64_t *a, *b, *w, *uw, *tf0, *ti0, *tf, *ti;
  int64_t *runc, *bc;
  uint64_t* bar;   // mbarriers: blocks, segments and boundary carries complete
  uint64_t* sent;  // exchanges that each CTA sent, at the end
  uint8_t* wd;
};

constexpr int kMinRun = 4;

__host__ __device__ inline size_t cluster_smem_words(int m, int C) {
  return 4 * (size_t)padded(m) + 2 * (size_t)m /* first pass */ + 2 * (size_t)m /* local passes */ +
         (size_t)m / kMinRun + 2 * (size_t)C + 3 + ((size_t)m + 7) / 8;
}

// One pass of the length-m transform on the block buffer.  Mode 0: forward, 1: inverse, 2: last
// forward pass, square and first inverse pass, 3: the last inverse pass, whose results go to the
// natural owners.  tw: this pass's twiddles, (r - 1) q + t for r >= 1.
template <int R, int Mode>
__device__ __forceinline__ void local_tasks(const Layout& S, int m, int span, const uint64_t* tw, uint32_t rank,
                                            int seg) {
  const int q = span / R, lq = __ffs(q) - 1, lseg = __ffs(seg) - 1;
  for (int task = threadIdx.x; task < m / R; task += blockDim.x) {
    const int t = task & (q - 1), off = (task >> lq) * span + t, b0 = sw(off);
    uint64_t v[R];
    lazy::W3 x[R];
#pragma unroll
    for (int d = 0; d < R; ++d) v[d] = S.b[task_pos<false>(b0, q, 0, d)];
    if constexpr (Mode == 0 || Mode == 2) {
      widen<R>(v, x);
      lazy::dif<R>(x, v);
    }
    if constexpr (Mode == 0) {
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = lazy::mul(v[r], tw[(r - 1) * q + t]);
    } else {
      if constexpr (Mode == 2) {
#pragma unroll
        for (int r = 0; r < R; ++r) x[r] = lazy::mul3(v[r], v[r]);
      } else {
        x[0] = lazy::from_word(v[0]);
#pragma unroll
        for (int r = 1; r < R; ++r) x[r] = lazy::mul3(v[r], tw[(r - 1) * q + t]);
      }
      lazy::dit_inv<R>(x, v);
    }
#pragma unroll
    for (int d = 0; d < R; ++d) {
      if constexpr (Mode == 3) {
        const int p = off + q * d;
        send(S.a + sw((int)rank * seg + (p & (seg - 1))), S.bar + 1, (uint32_t)(p >> lseg), v[d]);
      } else {
        S.b[task_pos<false>(b0, q, 0, d)] = v[d];
      }
    }
  }
}

template <int Mode>
__device__ __forceinline__ void local_pass(int R, const Layout& S, int m, int span, const uint64_t* tw,
                                           uint32_t rank, int seg) {
  if (R == 8) local_tasks<8, Mode>(S, m, span, tw, rank, seg);
  else if (R == 4) local_tasks<4, Mode>(S, m, span, tw, rank, seg);
  else local_tasks<2, Mode>(S, m, span, tw, rank, seg);
}

// Adds `carry` to a run of K digits held at s (the first K - 1 rebalance, the last absorbs).
__device__ __forceinline__ void carry_into_run(uint64_t* a, const uint8_t* wd, int i0, int K, int64_t carry,
                                               uint32_t& status) {
  for (int k = 0; k + 1 < K && carry != 0; ++k) {
    int64_t q;
    a[sw(i0 + k)] = (uint64_t)balance((int64_t)a[sw(i0 + k)] + carry, wd[i0 + k], q);
    carry = q;
  }
  if (carry != 0) {
    a[sw(i0 + K - 1)] = (uint64_t)((int64_t)a[sw(i0 + K - 1)] + carry);
    if (carry > kAbsorbLimit || carry < -kAbsorbLimit) status |= kStatusCarryOverflow;
  }
}

template <int C>
__global__ void __launch_bounds__(512) cluster_square_loop(const ClusterDesc* __restrict__ descs,
                                                             const __grid_constant__ ClusterDesc one, int pass_log2) {
  extern __shared__ __align__(16) uint64_t sm[];
  constexpr int kLogC = C == 4 ? 2 : (C == 8 ? 3 : 4);
  const ClusterDesc& D = descs ? descs[blockIdx.x / C] : one;
  const uint32_t rank = cluster_rank();
  const int n = (int)D.n, m = n / C, seg = m / C, lseg = __ffs(seg) - 1;
  const int tid = threadIdx.x, bd = blockDim.x;
  const Passes P = make_passes((int)D.log2n - kLogC, pass_log2);
  Layout S;
  S.a = sm;
  S.b = S.a + padded(m);
  S.w = S.b + padded(m);
  S.uw = S.w + padded(m);
  S.tf0 = S.uw + padded(m);
  S.ti0 = S.tf0 + m;
  S.tf = S.ti0 + m;
  S.ti = S.tf + m;
  S.runc = reinterpret_cast<int64_t*>(S.ti + m);
  S.bc = S.runc + m / kMinRun;
  S.bar = reinterpret_cast<uint64_t*>(S.bc + C);
  S.sent = S.bar + 3;
  S.wd = reinterpret_cast<uint8_t*>(S.sent + C);
  if (tid == 0) {
    for (int k = 0; k < 3; ++k)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(S.bar + k)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    expect_bytes(S.bar, 8u * (uint32_t)m);
    expect_bytes(S.bar + 1, 8u * (uint32_t)m);
    expect_bytes(S.bar + 2, 8u * (uint32_t)C);
  }

  // ---- tables and digits ----
  // natural word of local index i (segment k = i / seg): k m + rank seg + i mod seg
  auto word = [&](int i) { return (i >> lseg) * m + (int)rank * seg + (i & (seg - 1)); };
  for (int i = tid; i < m; i += bd) {
    const int j = word(i);
    uint64_t w, uw;
    if (D.w) {
      w = D.w[j];
      uw = D.uw[j];
    } else {
      // the two-pass plan's separable weights (TwoPassDesc): j = j1 + n1 j2
      const uint32_t j1 = (uint32_t)j & (D.n1 - 1), j2 = (uint32_t)j / D.n1;
      const ulonglong2 cw = D.colw[j1], rw = D.rowf[2 * j2], ru = D.rowf[2 * j2 + 1];
      const bool wrapped = D.colf[j1] + (uint32_t)rw.y >= D.n;
      const uint64_t p = gl::mul(cw.x, rw.x);
      w = wrapped ? p : gl::add(p, p);
      uw = gl::mul(cw.y, wrapped ? ru.y : ru.x);
    }
    S.w[sw(i)] = w;
    S.uw[sw(i)] = uw;
    S.wd[i] = D.widths[j];
    S.a[sw(i)] = (uint64_t)D.digits[j];
  }
  // first pass: omega_n^(t brev(r)), t = rank seg + u; local passes: omega_span^(t brev(r))
  for (int i = tid; i < m - seg; i += bd) {
    const int r = (i >> lseg) + 1, t = (int)rank * seg + (i & (seg - 1));
    const int e = t * brev_bits(r, kLogC);
    S.tf0[i] = D.pw[e];
    S.ti0[i] = D.pw[(n - e) & (n - 1)];
  }
  for (int j = 0, span = m, o = 0; j + 1 < P.m; ++j) {
    const int R = P.radix[j], q = span / R, lq = __ffs(q) - 1, bits = __ffs(R) - 1, scale = n / span;
    for (int i = tid; i < span - q; i += bd) {
      const int e = (i & (q - 1)) * brev_bits((i >> lq) + 1, bits) * scale;
      S.tf[o + i] = D.pw[e];
      S.ti[o + i] = D.pw[(n - e) & (n - 1)];
    }
    o += span - q;
    span = q;
  }
  uint32_t status = 0;
  const int K = D.short_runs ? 4 : 8, runs = m / K, lrps = __ffs(seg / K) - 1;
  for (int i = tid; i < runs; i += bd) S.runc[i] = 0;
  for (int i = tid; i < C; i += bd) S.bc[i] = 0;
  __syncthreads();
  if (D.carry) {
    // pending run carries of a two-pass state (runs of `tile` words)
    const int T = (int)D.tile;
    for (int i = tid; i < m / T; i += bd) {
      const uint32_t j = (uint32_t)word(i * T), j1 = j & (D.n1 - 1), r = j / D.n1, t = j1 / D.tile;
      const size_t pi = t > 0 ? (size_t)(t - 1) * D.n2 + r
                              : (size_t)(D.ntiles - 1) * D.n2 + (r ? r - 1 : D.n2 - 1);
      carry_into_run(S.a, S.wd, i * T, T, D.carry[pi], status);
    }
  }
  // every CTA of the cluster runs before any writes into another's shared memory, and every
  // pending carry is read before one is cleared at the end
  cluster_sync();

  // exchanges that this CTA sent, and that it received and re-armed, when it leaves the loop
  uint64_t sent = 0, passed = 0;
  bool lost = false;  // this CTA gave up
  const uint64_t stop = rank == 0 && D.quit_at < D.iterations ? D.quit_at : D.iterations;
  for (uint64_t it = 0; it < stop; ++it) {
    const bool um = D.unsigned_first && it == 0;
    // carry-in of the run before, then weight
    for (int i = tid; i < runs; i += bd) {
      const int64_t carry = (i & ((1 << lrps) - 1)) ? S.runc[i - 1] : S.bc[i >> lrps];
      carry_into_run(S.a, S.wd, i * K, K, carry, status);
#pragma unroll 4
      for (int k = 0; k < K; ++k) {
        uint64_t& v = S.a[sw(i * K + k)];
        v = lazy::mul_digit((int64_t)v, S.w[sw(i * K + k)]);
      }
    }
    if ((lost = gave_up(status))) {  // of the exchange before: no wait has run when it = 0
      sent = 3 * it;
      passed = sent - 1;
      break;
    }
    if (it && tid == 0) expect_bytes(S.bar + 2, 8u * (uint32_t)C);
    // radix-C pass: block r goes to CTA r
    for (int u = tid; u < seg; u += bd) {
      uint64_t v[C];
      lazy::W3 x[C];
#pragma unroll
      for (int k = 0; k < C; ++k) x[k] = lazy::from_word(S.a[sw(k * seg + u)]);
      lazy::dif<C>(x, v);
#pragma unroll
      for (int r = 1; r < C; ++r) v[r] = lazy::mul(v[r], S.tf0[(r - 1) * seg + u]);
#pragma unroll
      for (int r = 0; r < C; ++r) send(S.b + sw((int)rank * seg + u), S.bar, (uint32_t)r, v[r]);
    }
    const uint32_t parity = (uint32_t)it & 1u;
    await_phase(S.bar, parity, D.wait_ns, status);
    int span = m, o = 0;
    for (int j = 0; j + 1 < P.m && !lost; ++j) {
      local_pass<0>(P.radix[j], S, m, span, S.tf + o, rank, seg);
      o += span - span / P.radix[j];
      span /= P.radix[j];
      if (j) __syncthreads();
      else lost = gave_up(status);
    }
    if (lost) {
      sent = 3 * it + 1;
      passed = 3 * it;
      break;
    }
    if (tid == 0) expect_bytes(S.bar, 8u * (uint32_t)m);
    local_pass<2>(P.radix[P.m - 1], S, m, span, nullptr, rank, seg);
    __syncthreads();
    for (int j = P.m - 2; j > 0; --j) {
      o -= span * P.radix[j] - span;
      span *= P.radix[j];
      local_pass<1>(P.radix[j], S, m, span, S.ti + o, rank, seg);
      __syncthreads();
    }
    local_pass<3>(P.radix[0], S, m, m, S.ti, rank, seg);
    await_phase(S.bar + 1, parity, D.wait_ns, status);
    // inverse radix-C pass, in place on the segments
    for (int u = tid; u < seg; u += bd) {
      uint64_t v[C];
      lazy::W3 x[C];
      x[0] = lazy::from_word(S.a[sw(u)]);
#pragma unroll
      for (int r = 1; r < C; ++r) x[r] = lazy::mul3(S.a[sw(r * seg + u)], S.ti0[(r - 1) * seg + u]);
      lazy::dit_inv<C>(x, v);
#pragma unroll
      for (int k = 0; k < C; ++k) S.a[sw(k * seg + u)] = v[k];
    }
    if ((lost = gave_up(status))) {
      sent = 3 * it + 2;
      passed = 3 * it + 1;
      break;
    }
    if (tid == 0) expect_bytes(S.bar + 1, 8u * (uint32_t)m);
    // unweight and carry; a segment's last carry goes to the CTA that holds the next word
    for (int i = tid; i < runs; i += bd) {
      int64_t carry = (!D.prp && rank == 0 && i == 0) ? -2 : 0;
#pragma unroll 4
      for (int k = 0; k < K; ++k) {
        uint64_t& v = S.a[sw(i * K + k)];
        uint64_t y = lazy::mul(v, S.uw[sw(i * K + k)]);
        if (um) y = gl::canon(y);
        v = (uint64_t)carry_digit(y, um, carry, S.wd[i * K + k], carry);
      }
      S.runc[i] = carry;
      if (((i + 1) & ((1 << lrps) - 1)) == 0) {
        const int k = i >> lrps;
        if (rank + 1 < C) send(S.bc + k, S.bar + 2, rank + 1, (uint64_t)carry);
        else send(S.bc + ((k + 1) & (C - 1)), S.bar + 2, 0, (uint64_t)carry);
      }
    }
    __syncthreads();  // the CTA's own run carries
    await_phase(S.bar + 2, parity, D.wait_ns, status);
  }
  if (!lost) {
    if (stop < D.iterations) status |= kStatusClusterTimeout;
    lost = gave_up(status);
    sent = 3 * stop;
    passed = lost && sent ? sent - 1 : sent;
  }

  if (!lost) {
    for (int i = tid; i < runs; i += bd) {
      const int64_t carry = (i & ((1 << lrps) - 1)) ? S.runc[i - 1] : S.bc[i >> lrps];
      carry_into_run(S.a, S.wd, i * K, K, carry, status);
      for (int k = 0; k < K; ++k) D.digits[word(i * K + k)] = (int64_t)S.a[sw(i * K + k)];
    }
    if (D.carry)
      for (int i = tid; i < m / (int)D.tile; i += bd) D.carry[(size_t)rank * (m / (int)D.tile) + i] = 0;
  }
  if (status) atomicOr(D.status, status);
  // No CTA leaves while another may still store into its memory: past this barrier nothing more is
  // sent, and a CTA that gave up waits (with a limit) for the words on their way to it.  One that did
  // not give up has received all that was sent to it.
  if (tid < C) store_remote(S.sent + rank, (uint32_t)tid, sent);
  cluster_sync();
  if (lost && tid == 0) {
    for (int b = 0; b < 3; ++b) {
      const uint32_t missing = cluster::bytes_missing(b, passed, S.sent, rank, C, (uint32_t)m);
      if (missing) complete_bytes(S.bar + b, missing);
      uint32_t closing = 0;
      await_phase(S.bar + b, (uint32_t)(cluster::armed(passed, b) - 1) & 1u, D.wait_ns, closing);
    }
  }
}

template <int C>
cudaError_t launch_c(const ClusterDesc* descs, const ClusterDesc& one, uint32_t count, uint32_t max_n, int threads, int pass_log2,
                     cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(count * C);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = 8 * cluster_smem_words((int)max_n / C, C);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, cluster_square_loop<C>, descs, one, pass_log2);
}

// Clusters of C CTAs with the largest shared memory (and threads) that the device holds at once;
// 0 when it cannot launch them.  Raises the kernel's limits.  Once per device.
template <int C>
int max_clusters() {
  static std::mutex mu;
  static std::map<int, int> cache;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  std::lock_guard<std::mutex> lock(mu);
  auto it = cache.find(dev);
  if (it != cache.end()) return it->second;
  int count = 0;
  DeviceInfo info;
  const size_t smem = 8 * cluster_smem_words(2048, C);
  if (device_info(info) == cudaSuccess && smem <= (size_t)info.smem_per_block_optin &&
      cudaFuncSetAttribute(cluster_square_loop<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) ==
          cudaSuccess &&
      (C <= 8 || cudaFuncSetAttribute(cluster_square_loop<C>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
                     cudaSuccess)) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C);
    cfg.blockDim = dim3(512);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&count, cluster_square_loop<C>, &cfg) != cudaSuccess) count = 0;
  }
  cudaGetLastError();
  return cache[dev] = count;
}

}  // namespace

namespace {
bool cluster_fits(uint32_t n, uint32_t C) {
  // segments hold whole 8-word runs, blocks at least two passes and at most 2048 words
  return n >= 8 * C * C && n / C >= 64 && n / C <= 2048;
}

int cluster_max_active(uint32_t C) { return C == 4 ? max_clusters<4>() : (C == 8 ? max_clusters<8>() : max_clusters<16>()); }
}  // namespace

// One B200, us a squaring of one test alone, against the resident (to 4096) or two-pass kernels:
//   n        512    1024    2048    4096    8192   16384   32768
//   before  5.12    6.52    8.26    14.1    15.9    17.3    18.6
//   C = 4   4.42    4.57    5.46    6.81    10.0     -       -
//   C = 8   4.54    5.00    5.09    5.88    7.14    10.2     -
//   C = 16   -       -      7.20    7.29    8.01    9.17    11.8
//   now     4.05    4.13    4.68    5.54    6.86    8.53    11.1   (the size taken; the rows above are older)
// About 4 us are the latency of a dozen phases of one or two warps per scheduler.  Local passes of
// radix 4 beat radix 8 (half as long for two of the three stages) up to blocks of 1024 words.
// A launch of several tests takes the largest size of which the GPU holds all clusters at once; where
// it does not even for C = 4, one CTA per test (lnt_resident.cu) does more squarings a second.
ClusterChoice cluster_choice(uint32_t min_n, uint32_t max_n, uint32_t count) {
  ClusterChoice c;
  for (uint32_t C = max_n <= 1024 ? 4 : (max_n <= 8192 ? 8 : 16); C >= 4; C /= 2) {
    if (!cluster_fits(min_n, C) || !cluster_fits(max_n, C) || cluster_max_active(C) < (int)count) continue;
    const int m = (int)(max_n / C);
    c.size = C;
    c.threads = std::max(64, std::min({m / 2, std::max(256, m / 4), 512}));
    c.pass_log2 = m >= 2048 ? 3 : 2;
    break;
  }
  return c;
}

cudaError_t launch_cluster(const ClusterDesc* descs, const ClusterDesc& one, uint32_t count, uint32_t max_n, uint32_t C, int threads,
                           int pass_log2, cudaStream_t s) {
  switch (C) {
    case 4: return launch_c<4>(descs, one, count, max_n, threads, pass_log2, s);
    case 8: return launch_c<8>(descs, one, count, max_n, threads, pass_log2, s);
    case 16: return launch_c<16>(descs, one, count, max_n, threads, pass_log2, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace lnt
