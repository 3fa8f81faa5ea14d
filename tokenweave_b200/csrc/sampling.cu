// Token sampling from fp32 logits in ONE launch for the whole batch: temperature, top-k, top-p, min-p
// and the random draw, one cluster of CTAs per row, no sort and no host round trip.
//
// The reference samples with a full sort of every row plus softmax / cumsum / scatter passes and one
// generator call per seeded request (vllm/v1/sample/ops/topk_topp_sampler.py:170-262,
// vllm/v1/sample/sampler.py:17-270). Here the support is described by ONE threshold on the scaled
// logit: the k-th largest value comes from a radix select on the float bits (counts), the top-p boundary from
// a radix select weighted by exp(x - max) (the smallest value whose ascending cumulative mass exceeds
// 1 - top_p, the reference's rule), min-p is max + log(min_p).
// The draw is the Gumbel / exponential race argmax(x_i + g_i) over the kept set, with g_i from a
// counter-based generator keyed by (row seed, token index), so a seeded request repeats exactly.
//
// A row has a cluster of 1 to 8 CTAs, as many as the SMs have room for at once, each with a part of it (in shared memory where
// that fits, else read again from L2). With top-k up to the thread count, the k-th largest of the threads' maxima bounds what can
// be kept from below: the few elements that reach it go to rank 0, which does everything else with them. Otherwise the selects
// run over the cluster: each CTA counts its part, adds its occupied counters to those of rank 0 through distributed shared
// memory, and rank 0 looks the digit up. The digits have 11, 11 and 10 bits, so the first one (sign, exponent, two bits of
// mantissa) spreads logits over enough counters that few lanes of a warp meet at one. Masses are integers of 64 bits, units of
// 2^-40 of the largest: shared memory has no atomics for floats without retries, and an integer sum does not depend on the order.
// 144 rows of 128256 logits, us: 32 with top-k, 43 with top-k and top-p, 115 with top-p alone, 46 without; 133 mixed (1215 with one
// CTA per row, digits of 8 bits and atomics on floats). Reading the logits takes 11; a further pass over L2 takes about as long,
// the rest is the atomics of the first digit.
#include "tw_common.cuh"
#include "tw_host.h"
#include "tw_kernels.h"

namespace tw {

constexpr int SAMPLE_THREADS = 1024;

struct SampleRowParams {   // one per row, 32 bytes
  float temperature;       // <= 0: greedy
  int top_k;               // <= 0 or >= V: disabled
  float top_p;             // >= 1: disabled
  float min_p;             // <= 0: disabled
  unsigned long long seed;
  unsigned long long pad;
};

__device__ __forceinline__ uint32_t sortable_key(float x) {
  const uint32_t u = __float_as_uint(x);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ float gumbel_noise(unsigned long long seed, int i) {
  unsigned long long z = seed + 0x9E3779B97F4A7C15ull * static_cast<unsigned long long>(i + 1);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  const float u = (static_cast<float>(z >> 40) + 0.5f) * (1.0f / 16777216.0f);   // (0, 1)
  return -__logf(-__logf(u));
}

constexpr int SAMPLE_BINS = 2048;
constexpr int SAMPLE_MAX_CLUSTER = 8;
constexpr int SAMPLE_MAX_CANDIDATES = 4096;
constexpr int SAMPLE_SMEM_MAX = 220 * 1024;

struct alignas(16) SampleShared {
  unsigned int count[SAMPLE_BINS];         // this CTA's counters: counts, or the upper words of masses
  unsigned int low[SAMPLE_BINS];           // the lower words of masses
  unsigned long long total[SAMPLE_BINS];   // rank 0: those of the cluster
  float cand[SAMPLE_MAX_CANDIDATES];       // rank 0: what top-k can keep, and where it stands in the row
  int cand_at[SAMPLE_MAX_CANDIDATES];
  unsigned long long warp_sums[32];
  unsigned long long left;                 // what is left to count or to weigh inside the digit found so far
  float max_of[SAMPLE_MAX_CLUSTER];        // maxima, and then in rank 0 the best of the draw, of every rank
  int best_of[SAMPLE_MAX_CLUSTER];
  uint32_t bound_of[SAMPLE_MAX_CLUSTER];
  float scratch[32];
  int scratch_i[32];
  uint32_t prefix;
  unsigned int candidates;
};

__device__ __forceinline__ uint32_t smem_at_rank(const void* p, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_barrier() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t ld_rank_u32(const void* p, uint32_t rank) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(smem_at_rank(p, rank)) : "memory");
  return v;
}
__device__ __forceinline__ void st_rank_u32(void* p, uint32_t rank, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(smem_at_rank(p, rank)), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t add_rank_u32(void* p, uint32_t rank, uint32_t v) {
  uint32_t old;
  asm volatile("atom.relaxed.cluster.shared::cluster.add.u32 %0, [%1], %2;"
               : "=r"(old) : "r"(smem_at_rank(p, rank)), "r"(v) : "memory");
  return old;
}
__device__ __forceinline__ void add_rank_u64(void* p, uint32_t rank, unsigned long long v) {
  asm volatile("red.relaxed.cluster.shared::cluster.add.u64 [%0], %1;" ::"r"(smem_at_rank(p, rank)), "l"(v) : "memory");
}

// A CTA's part of a row, or the list of candidates: `each` runs over what this thread takes of it, scaled.
struct RowPart {
  const float* src;
  float scale;               // 1 where src is the shared copy
  int n, n4;                 // elements, and fours of them that can be loaded at once
  template <typename F>
  __device__ __forceinline__ void four(const float4& v, int i, F& f) const {
    f(v.x * scale, 4 * i);
    f(v.y * scale, 4 * i + 1);
    f(v.z * scale, 4 * i + 2);
    f(v.w * scale, 4 * i + 3);
  }
  template <typename F>
  __device__ __forceinline__ void each(F f) const {
    const float4* src4 = reinterpret_cast<const float4*>(src);
    constexpr int AHEAD = 4;             // loads in flight per thread: 64 KB per CTA cover the latency of L2
    int i = threadIdx.x;
    for (; i + (AHEAD - 1) * SAMPLE_THREADS < n4; i += AHEAD * SAMPLE_THREADS) {
      float4 v[AHEAD];
#pragma unroll
      for (int a = 0; a < AHEAD; ++a) v[a] = src4[i + a * SAMPLE_THREADS];
#pragma unroll
      for (int a = 0; a < AHEAD; ++a) four(v[a], i + a * SAMPLE_THREADS, f);
    }
    for (; i < n4; i += SAMPLE_THREADS) four(src4[i], i, f);
#pragma unroll 4
    for (i = 4 * n4 + threadIdx.x; i < n; i += SAMPLE_THREADS) f(src[i] * scale, i);
  }
};

// exp(x - m) in units of 2^-40; the maximum itself counts one, also where it is infinite, and a NaN nothing
__device__ __forceinline__ unsigned long long mass_of(float x, float m) {
  const float e = x == m ? 1.f : __expf(x - m);
  return e > 0.f ? __float2ull_rn(fminf(e, 1.f) * 1099511627776.f) : 0ull;
}
// to a counter of 64 bits as two words, with the carry: shared memory adds words in one go, wider integers with retries
__device__ __forceinline__ void add_mass(unsigned int* low, unsigned int* high, unsigned long long v) {
  const unsigned int lo = static_cast<unsigned int>(v);
  unsigned int hi = static_cast<unsigned int>(v >> 32);
  if (lo != 0 && atomicAdd(low, lo) > ~lo) ++hi;
  if (hi != 0) atomicAdd(high, hi);
}

__device__ __forceinline__ void best_pair(float& v, int& i, float ov, int oi) {
  if (ov > v || (ov == v && oi < i)) {
    v = ov;
    i = oi;
  }
}

// The digit in which `left` runs out - counting from the largest digit down (counts), or from the smallest up (masses) -, appended
// to the prefix of every rank, and what is left inside it. Masses that never run out end in the largest occupied digit, and so below.
template <bool MASS>
__device__ __forceinline__ void find_digit(SampleShared& s, int shift, int ranks) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned long long left = s.left;
  const unsigned long long h0 = s.total[2 * tid], h1 = s.total[2 * tid + 1];
  unsigned long long incl = h0 + h1;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) s.warp_sums[warp] = incl;
  int last = h1 != 0 ? 2 * tid + 1 : h0 != 0 ? 2 * tid : -1;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) last = max(last, __shfl_xor_sync(0xffffffffu, last, o));
  if (lane == 0) s.scratch_i[warp] = last;
  __syncthreads();
  unsigned long long before = 0, all = 0;
  for (int w = 0; w < 32; ++w) {
    const unsigned long long v = s.warp_sums[w];
    if (w < warp) before += v;
    all += v;
    last = max(last, s.scratch_i[w]);
  }
  const unsigned long long e0 = before + incl - h0 - h1, e1 = e0 + h0;
  int digit = -1;
  unsigned long long now = 0;
  if (MASS) {
    if (e0 <= left && e0 + h0 > left) digit = 2 * tid, now = left - e0;
    else if (e1 <= left && e1 + h1 > left) digit = 2 * tid + 1, now = left - e1;
    else if (left >= all && tid == 0) digit = max(last, 0), now = ~0ull;
  } else {
    if (all - e0 >= left && all - e0 - h0 < left) digit = 2 * tid, now = left - (all - e0 - h0);
    else if (all - e1 >= left && all - e1 - h1 < left) digit = 2 * tid + 1, now = left - (all - e1 - h1);
  }
  if (digit >= 0) {
    const uint32_t prefix = s.prefix | (static_cast<uint32_t>(digit) << shift);
    s.left = now;                          // only this CTA counts on
    if (ranks == 1) s.prefix = prefix;
    else
      for (int r = 0; r < ranks; ++r) st_rank_u32(&s.prefix, r, prefix);
  }
}

// The radix select: s.left is what to count on entry (rank 0), the key found is returned to all. MASS: the keys from tau on,
// by mass, s.left then being `share` of their total. ALONE: one CTA over a list of its own, else the cluster over the row.
template <bool MASS, bool ALONE>
__device__ __forceinline__ uint32_t select_key(SampleShared& s, const RowPart& x, float m, uint32_t tau, double share,
                                               uint32_t rank, int ranks) {
  const int tid = threadIdx.x;
  __syncthreads();
  if (tid == 0) s.prefix = 0u;
  for (int level = 0; level < 3; ++level) {
    const int shift = level == 0 ? 21 : level == 1 ? 10 : 0;
    const uint32_t digits = level == 2 ? 1023u : 2047u;
    const uint32_t mask = level == 0 ? 0u : 0xffffffffu << (shift + (level == 1 ? 11 : 10));
    s.count[tid] = s.count[tid + SAMPLE_THREADS] = 0u;
    if (MASS) s.low[tid] = s.low[tid + SAMPLE_THREADS] = 0u;
    if (!ALONE && rank == 0) s.total[2 * tid] = s.total[2 * tid + 1] = 0;
    if (ALONE) __syncthreads();
    else cluster_barrier();                // counters are clear everywhere, the last digit has arrived
    const uint32_t prefix = s.prefix;
    x.each([&](float xi, int) {
      const uint32_t key = sortable_key(xi);
      if (key < tau || (key & mask) != prefix) return;
      const uint32_t d = (key >> shift) & digits;
      if (MASS) add_mass(&s.low[d], &s.count[d], mass_of(xi, m));
      else atomicAdd(&s.count[d], 1u);
    });
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      unsigned long long v = s.count[2 * tid + j];
      if (MASS) v = (v << 32) + s.low[2 * tid + j];
      if (ALONE || ranks == 1) s.total[2 * tid + j] = v;
      else if (v != 0) add_rank_u64(&s.total[2 * tid + j], 0, v);
    }
    if (!ALONE) cluster_barrier();
    if (ALONE || rank == 0) {
      if (MASS && level == 0) {
        unsigned long long all = s.total[2 * tid] + s.total[2 * tid + 1];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) all += __shfl_xor_sync(0xffffffffu, all, o);
        if ((tid & 31) == 0) s.warp_sums[tid >> 5] = all;
        __syncthreads();
        if (tid == 0) {
          unsigned long long z = 0;
          for (int w = 0; w < 32; ++w) z += s.warp_sums[w];
          s.left = static_cast<unsigned long long>(share * static_cast<double>(z));
        }
        __syncthreads();
      }
      find_digit<MASS>(s, shift, ALONE ? 1 : ranks);
    }
  }
  if (ALONE) __syncthreads();
  else cluster_barrier();
  return s.prefix;
}

// The draw over one CTA's elements: argmax of x_i + gumbel_i over the keys from tau on (plain argmax when greedy), lowest index on
// ties. Warp 0 has the result.
template <typename At>
__device__ __forceinline__ void draw(SampleShared& s, const RowPart& x, uint32_t tau, bool greedy, unsigned long long seed, At at,
                                     float& best, int& best_i) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  best = -INFINITY;
  best_i = 0x7fffffff;
  x.each([&](float xi, int i) {
    if (sortable_key(xi) < tau) return;
    const int t = at(i);
    best_pair(best, best_i, greedy ? xi : xi + gumbel_noise(seed, t), t);
  });
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    best_pair(best, best_i, __shfl_xor_sync(0xffffffffu, best, o), __shfl_xor_sync(0xffffffffu, best_i, o));
  __syncthreads();
  if (lane == 0) {
    s.scratch[warp] = best;
    s.scratch_i[warp] = best_i;
  }
  __syncthreads();
  if (warp == 0) {
    best = s.scratch[lane];
    best_i = s.scratch_i[lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      best_pair(best, best_i, __shfl_xor_sync(0xffffffffu, best, o), __shfl_xor_sync(0xffffffffu, best_i, o));
  }
}

__global__ void __launch_bounds__(SAMPLE_THREADS, 1)
sample_kernel(const float* __restrict__ logits, long long ld, int V, int per, bool staged, int ranks,
              const SampleRowParams* __restrict__ params, int* __restrict__ out) {
  extern __shared__ uint8_t smem_raw[];
  SampleShared& s = *reinterpret_cast<SampleShared*>(smem_raw);
  float* slice = reinterpret_cast<float*>(smem_raw + sizeof(SampleShared));

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int row = blockIdx.x / ranks;
  const uint32_t rank = blockIdx.x % ranks;
  const SampleRowParams p = params[row];
  const bool greedy = !(p.temperature > 0.f);
  const float inv_t = greedy ? 1.f : 1.f / p.temperature;
  const int first = static_cast<int>(rank) * per;
  const int n = max(0, min(per, V - first));
  const float* src = logits + row * ld + first;

  // the part of the row - scaled into shared memory where it fits -, its maximum and the largest key of every thread
  float m = -INFINITY;
  uint32_t top = 0u;
  RowPart x{src, inv_t, n, (reinterpret_cast<uintptr_t>(src) & 15) == 0 ? n / 4 : 0};
  x.each([&](float v, int i) {
    if (staged) slice[i] = v;
    m = fmaxf(m, v);
    top = max(top, sortable_key(v));
  });
  if (staged) x = RowPart{slice, 1.f, n, n / 4};
  const bool by_k = !greedy && p.top_k > 0 && p.top_k < V, by_p = !greedy && p.top_p < 1.f, by_min = !greedy && p.min_p > 0.f;
  const double share = static_cast<double>(1.f - p.top_p);
  uint32_t tau = 0u;                       // keep keys >= tau
  float best;
  int best_i;
  if (tid == 0) s.candidates = 0u;
  cluster_barrier();                       // every CTA of the cluster runs: its shared memory may be written

  if (by_k && p.top_k <= SAMPLE_THREADS) {
    // The k-th largest of the threads' maxima is no larger than the k-th largest of the row: only what reaches it (22 bits of
    // it, in the CTA where it is highest) can be kept. That is little more than k elements, and rank 0 does the rest with them.
    if (tid == 0) {
      s.left = p.top_k;
      s.prefix = 0u;
    }
    for (int level = 0; level < 2; ++level) {
      const int shift = level == 0 ? 21 : 10;
      s.count[tid] = s.count[tid + SAMPLE_THREADS] = 0u;
      __syncthreads();
      if (level == 0 || (top >> 21) == (s.prefix >> 21)) atomicAdd(&s.count[(top >> shift) & 2047u], 1u);
      __syncthreads();
      s.total[2 * tid] = s.count[2 * tid];
      s.total[2 * tid + 1] = s.count[2 * tid + 1];
      find_digit<false>(s, shift, 1);
      __syncthreads();
    }
    uint32_t bound = s.prefix;
    if (ranks > 1) {
      if (tid < ranks) st_rank_u32(&s.bound_of[rank], tid, bound);
      cluster_barrier();
      for (int r = 0; r < ranks; ++r) bound = max(bound, s.bound_of[r]);
    }
    x.each([&](float v, int i) {
      if (sortable_key(v) < bound) return;
      const uint32_t at = ranks > 1 ? add_rank_u32(&s.candidates, 0, 1u) : atomicAdd(&s.candidates, 1u);
      if (at < SAMPLE_MAX_CANDIDATES) {
        st_rank_u32(&s.cand[at], 0, __float_as_uint(v));
        st_rank_u32(&s.cand_at[at], 0, static_cast<uint32_t>(first + i));
      }
    });
    cluster_barrier();
    if (tid == 0 && rank != 0) s.candidates = ld_rank_u32(&s.candidates, 0);
    cluster_barrier();                     // nobody else reaches into rank 0 from here on
    const int found = static_cast<int>(s.candidates);
    if (found <= SAMPLE_MAX_CANDIDATES) {
      if (rank != 0) return;
      const RowPart c{s.cand, 1.f, found, found / 4};
      if (tid == 0) s.left = p.top_k;
      tau = select_key<false, true>(s, c, 0.f, 0u, 0.0, 0, 1);
      if (by_p || by_min) {
        m = -INFINITY;
        c.each([&](float v, int) { m = fmaxf(m, v); });
        m = warp_max(m);
        if (lane == 0) s.scratch[warp] = m;
        __syncthreads();
        m = warp_max(s.scratch[lane]);
      }
      if (by_p) tau = max(tau, select_key<true, true>(s, c, m, tau, share, 0, 1));
      if (by_min) tau = max(tau, sortable_key(m + __logf(p.min_p)));
      const int* where = s.cand_at;
      draw(s, c, tau, false, p.seed, [=](int i) { return where[i]; }, best, best_i);
      if (tid == 0) out[row] = (best_i == 0x7fffffff) ? 0 : best_i;
      return;
    }
  }

  if (by_p || by_min) {
    m = warp_max(m);
    if (lane == 0) s.scratch[warp] = m;
    __syncthreads();
    m = warp_max(s.scratch[lane]);
    if (ranks > 1) {
      if (tid < ranks) st_rank_u32(&s.max_of[rank], tid, __float_as_uint(m));
      cluster_barrier();
      for (int r = 0; r < ranks; ++r) m = fmaxf(m, s.max_of[r]);
    }
  }
  if (by_k) {                              // more than a thousand, or thousands of equal ones
    if (tid == 0) s.left = p.top_k;
    tau = select_key<false, false>(s, x, m, 0u, 0.0, rank, ranks);
  }
  if (by_p) tau = max(tau, select_key<true, false>(s, x, m, tau, share, rank, ranks));
  // min-p comes last, as in the reference: p_i >= min_p * p_max  <=>  x_i >= max + log(min_p)
  if (by_min) tau = max(tau, sortable_key(m + __logf(p.min_p)));

  draw(s, x, tau, greedy, p.seed, [=](int i) { return first + i; }, best, best_i);
  cluster_barrier();                       // every rank has read the maxima
  if (ranks > 1) {
    if (tid == 0) {
      st_rank_u32(&s.max_of[rank], 0, __float_as_uint(best));
      st_rank_u32(&s.best_of[rank], 0, static_cast<uint32_t>(best_i));
    }
    cluster_barrier();
  }
  if (rank == 0 && tid == 0) {
    for (int r = 1; r < ranks; ++r) best_pair(best, best_i, s.max_of[r], s.best_of[r]);
    out[row] = (best_i == 0x7fffffff) ? 0 : best_i;
  }
}

}  // namespace tw

using namespace tw;

// params: `rows` records of 32 bytes {float temperature, int top_k, float top_p, float min_p, u64 seed, u64 pad}.
extern "C" int tw_sample(const float* logits, long long ld, int rows, int V, const void* params, int* out,
                         cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (V <= 0) {
    set_last_error("sample: empty vocabulary");
    return 1;
  }
  // As many CTAs per row as the SMs have room for at once, of at least 2048 logits each: what they share costs a few barriers
  // of the cluster, a second wave of CTAs costs more than longer parts.
  const int sms = device_sm_count();
  int ranks = 1;
  while (ranks < SAMPLE_MAX_CLUSTER && static_cast<long long>(rows) * ranks * 2 <= sms && V / (ranks * 2) >= 2048) ranks *= 2;
  const int per = ((V + ranks - 1) / ranks + 3) / 4 * 4;
  int smem = static_cast<int>(sizeof(SampleShared));
  const bool staged = static_cast<long long>(per) * 4 + smem <= SAMPLE_SMEM_MAX;
  if (staged) smem += per * 4;
  static thread_local int configured_dev = -1;
  int dev = 0;
  cudaGetDevice(&dev);
  if (configured_dev != dev) {
    cudaError_t e = cudaFuncSetAttribute(sample_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SAMPLE_SMEM_MAX);
    if (e != cudaSuccess) {
      set_last_error("cudaFuncSetAttribute(smem) failed: %s", cudaGetErrorString(e));
      return 1;
    }
    configured_dev = dev;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(rows) * ranks);
  cfg.blockDim = dim3(SAMPLE_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ranks;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, sample_kernel, logits, ld, V, per, staged, ranks,
                                     reinterpret_cast<const SampleRowParams*>(params), out);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_last_error("sample launch failed: %s", cudaGetErrorString(e));
    return 1;
  }
  return 0;
}
