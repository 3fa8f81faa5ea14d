// Products with few rows (decode steps, language-model heads): C[M,N] = A[M,K] * W[N,K]^T for M up to a few hundred.
//
// Such a product is bound by reading W once from memory, so the tile follows W and not A: 128 rows of W (64 gate and 64 up
// rows of a gated product) are the M side of tcgen05.mma, and ALL rows of A, padded to 16, are its N side. A stage of the
// pipeline is then 16 KB of weights and M x 128 bytes of activations, where a tile of 128 rows of A would fill two thirds of
// it with padding, and a narrow N (4096 outputs are 32 tiles) is spread over the chip by cutting K: a thread-block cluster of
// up to 8 CTAs shares a tile, each CTA sums its part of K in TMEM, and the parts are added through distributed shared memory
// in the order of the ranks - no workspace in global memory, no counters, the same result on every run.
//
//   warp 0      TMA producer (weights with an evict-first policy: they are read once)
//   warp 1      MMA issuer
//   warps 2..5  accumulators TMEM -> shared memory (fp32, where the stages were), then all threads of the cluster add the
//               parts and run the epilogue on 8 outputs of one row each
// What bounds it: memory. The down projection 4096x14336 of 48 rows takes 27 us (4.4 TB/s; 62 us with tiles of 128 rows of A,
// which are 32 CTAs), a head of 128256x4096 164 us (6.4 TB/s), the gated 2x14336x4096 43 us (5.5 TB/s; before 67 us).
// Launched to start while the kernel before it still runs: a step of 77 short kernels takes 937 us instead of 963.
// TMEM is given back before a CTA waits for the others of its cluster, so waiting for it never waits for a cluster.
// Every mbarrier wait is bounded; after a timeout the CTA still takes part in the cluster's barriers.
#include "tw_common.cuh"
#include "tw_host.h"
#include "tw_kernels.h"
#include "tw_pair.cuh"

namespace tw {

constexpr int SK_ROWS = 128;            // rows of W per tile
constexpr int SK_THREADS = 192;
constexpr int SK_MAX_STAGES = 16;
constexpr int SK_MAX_TOKENS = 256;
constexpr int SK_W_BYTES = SK_ROWS * 128;   // a k-block is 128 bytes of every row: 64 bf16 or 128 e4m3

struct SkinnyParams {
  __nv_bfloat16* C;
  float* logits;            // instead of C: the same numbers (rounded to bf16), in fp32 and times logit_scale
  float logit_scale;
  long long ldc;
  const __nv_bfloat16* bias;
  const float* row_scale;
  const float* col_scale;   // fp8: per-output-channel scale (may be null)
  int M, N;
  int num_kb;
  int tn;                   // rows of A, padded to 16
  int stages;
  int dump_rows;            // rows of A whose sums are in shared memory at once (all where K is cut)
  int split;                // CTAs of a cluster: parts of K
  int tmem_cols;
  int up_row_offset;
  GemmActs acts;
  uint32_t* status;
};

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t local_addr, uint32_t rank) {
  float4 v;
  asm volatile(
      "{\n\t.reg .u32 a;\n\tmapa.shared::cluster.u32 a, %4, %5;\n\t"
      "ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [a];\n\t}"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
      : "r"(local_addr), "r"(rank)
      : "memory");
  return v;
}

template <bool GLU, bool FP8, int KBS, bool PAIR>
__global__ void __launch_bounds__(SK_THREADS, 2)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmW, const SkinnyParams p) {
  constexpr int BK = FP8 ? 128 : 64;
  constexpr int OUT = GLU ? SK_ROWS / 2 : SK_ROWS;      // output columns per tile
  constexpr int CTAS = PAIR ? 2 : 1;                    // that share a tile's MMAs: each brings 128 rows of W and its share of A's
  const int a_rows = p.tn / CTAS;
  const int kb_bytes = SK_W_BYTES + a_rows * 128;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  __shared__ uint64_t full_bar[SK_MAX_STAGES], empty_bar[SK_MAX_STAGES], acc_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = CTAS * p.split > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const int part = rank / CTAS, half = rank % CTAS;
  const int w0 = (blockIdx.x / (CTAS * p.split) * CTAS + half) * OUT;   // first row of W and output column
  const int kb0 = static_cast<int>(static_cast<long long>(p.num_kb) * part / p.split);
  const int kb1 = static_cast<int>(static_cast<long long>(p.num_kb) * (part + 1) / p.split);

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&acc_bar, 1);
    abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmW);
  }
  allow_dependents();
  if (warp == 0 && elect_one()) {           // the first stages' weights on their way to L2 while the kernel before still runs
    const int ahead = min(kb1, kb0 + p.stages * KBS);
    for (int kb = kb0; kb < ahead; ++kb) {
      tma_prefetch_2d(&tmW, kb * BK, w0);
      if (GLU) tma_prefetch_2d(&tmW, kb * BK, w0 + p.up_row_offset);
    }
  }
  wait_predecessor();
  if (PAIR) {
    __syncthreads();
    cluster_sync_all();                     // both CTAs' barriers exist before anyone signals across
  }
  if (warp == 1) {
    if (PAIR) {
      tmem_alloc_pair(&tmem_slot, p.tmem_cols);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(&tmem_slot, p.tmem_cols);
      tmem_relinquish();
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = tmem_slot;

  // One thread of each issuing warp, chosen by elect.sync and not by its lane number: the compiler then knows that a single
  // thread runs the loop, and one CTA gets through a k-block in 0.17 us instead of 0.31.
  if (warp == 0) {
    if (elect_one()) {
      const uint64_t once = policy_evict_first();
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; kb += KBS) {
        if (!mbar_wait(&empty_bar[stage], phase ^ 1)) {
          report_error(p.status, TW_ERR_MBAR_TIMEOUT);
          abort_flag = 1;
          break;
        }
        uint8_t* sw = smem + stage * KBS * kb_bytes;
        const uint32_t full = PAIR ? map_to_cta(smem_u32(&full_bar[stage]), rank & ~1) : 0u;   // the leader's
        if (half == 0) mbar_expect_tx(&full_bar[stage], CTAS * KBS * kb_bytes);
        auto load_w = [&](uint8_t* dst, int x, int y) {
          if (PAIR) tma_load_2d_pair_hint(dst, &tmW, full, x, y, once);
          else tma_load_2d_hint(dst, &tmW, &full_bar[stage], x, y, once);
        };
#pragma unroll
        for (int h = 0; h < KBS; ++h, sw += kb_bytes) {
          const int x = min(kb + h, kb1) * BK;    // past the part's end: loaded, not multiplied (past K: zeros)
          load_w(sw, x, w0);
          if (GLU) load_w(sw + SK_W_BYTES / 2, x, w0 + p.up_row_offset);
          if (PAIR) tma_load_2d_pair(sw + SK_W_BYTES, &tmA, full, x, half * a_rows);
          else tma_load_2d(sw + SK_W_BYTES, &tmA, &full_bar[stage], x, 0);
        }
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    if (half == 0 && elect_one()) {
      const uint32_t idesc = FP8 ? make_idesc_e4m3(CTAS * SK_ROWS, p.tn) : make_idesc_bf16(CTAS * SK_ROWS, p.tn, 0, 0);
      auto commit = [&](uint64_t* bar) {    // to both CTAs of a pair
        if (PAIR) {
          umma_commit_pair(map_to_cta(smem_u32(bar), rank));
          umma_commit_pair(map_to_cta(smem_u32(bar), rank + 1));
        } else {
          umma_commit(bar);
        }
      };
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; kb += KBS) {
        if (!mbar_wait(&full_bar[stage], phase)) {
          report_error(p.status, TW_ERR_MBAR_TIMEOUT);
          abort_flag = 1;
          break;
        }
        tc_fence_after_sync();
        const uint32_t sw = smem_u32(smem + stage * KBS * kb_bytes);
#pragma unroll
        for (int h = 0; h < KBS; ++h) {
          if (KBS > 1 && kb + h >= kb1) break;
          const uint64_t w_desc = make_smem_desc_sw128(sw + h * kb_bytes, 16, 1024);
          const uint64_t a_desc = make_smem_desc_sw128(sw + h * kb_bytes + SK_W_BYTES, 16, 1024);
#pragma unroll
          for (int k = 0; k < 4; ++k) {     // 32 bytes further along K: +2 in the descriptor's 16-byte units
            const uint32_t acc = (kb != kb0 || h != 0 || k != 0) ? 1u : 0u;
            if (PAIR && FP8) umma_ss_pair_f8(tmem, w_desc + 2 * k, a_desc + 2 * k, idesc, acc);
            else if (PAIR) umma_ss_pair(tmem, w_desc + 2 * k, a_desc + 2 * k, idesc, acc);
            else if (FP8) umma_ss_f8(tmem, w_desc + 2 * k, a_desc + 2 * k, idesc, acc);
            else umma_ss(tmem, w_desc + 2 * k, a_desc + 2 * k, idesc, acc);
          }
        }
        commit(&empty_bar[stage]);
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
      commit(&acc_bar);
    }
  } else if (!mbar_wait(&acc_bar, 0)) {
    report_error(p.status, TW_ERR_MBAR_TIMEOUT);
    abort_flag = 1;
  }
  __syncthreads();
  if (abort_flag) {                         // copies in flight land before shared memory is reused or released
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
  }

  const uint32_t part0 = smem_u32(smem);
  constexpr int GROUPS = OUT / 8;
  for (int t0 = 0; t0 < p.tn; t0 += p.dump_rows) {
    const int t1 = min(t0 + p.dump_rows, p.tn);
    if (warp >= 2) {
      // accumulators -> shared memory, [row of A][row of W]: lanes are rows of W, so a warp writes 128 bytes in a row
      tc_fence_after_sync();
      const int q = warp & 3;
      float* dst = reinterpret_cast<float*>(smem) + q * 32 + lane;
      const uint32_t src = tmem + (static_cast<uint32_t>(q * 32) << 16);
      if (!abort_flag) {
#pragma unroll 1
        for (int c = t0; c < t1; c += 16) {
          uint32_t v[16];
          tmem_ld_32x16(src + c, v);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 16; ++j) dst[(c - t0 + j) * SK_ROWS] = __uint_as_float(v[j]);
        }
      }
      tc_fence_before_sync();
    }
    __syncthreads();
    if (warp == 1 && t1 == p.tn) {
      tc_fence_after_sync();
      if (PAIR) tmem_dealloc_pair(tmem, p.tmem_cols);
      else tmem_dealloc(tmem, p.tmem_cols);
    }
    if (p.split > 1) {
      __syncwarp();
      cluster_sync_all();
    }

    // ---- sums of the parts and epilogue: 8 neighbouring outputs of one row at a time ----
    const int items = (min(t1, p.M) - t0) * GROUPS;
    for (int i = part * SK_THREADS + threadIdx.x; i < items; i += p.split * SK_THREADS) {
      const int row = i / GROUPS, g = i % GROUPS;
      const int t = t0 + row, n = w0 + g * 8;
      if (n >= p.N) continue;
      float v[8], u[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = u[e] = 0.f;
      const uint32_t at = part0 + (row * SK_ROWS + g * 8) * 4;
      for (int s = 0; s < p.split; ++s) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float4 a;
          if (p.split > 1) a = ld_cluster_f4(at + h * 16, s * CTAS + half);
          else a = *reinterpret_cast<const float4*>(smem + (row * SK_ROWS + g * 8) * 4 + h * 16);
          v[4 * h] += a.x; v[4 * h + 1] += a.y; v[4 * h + 2] += a.z; v[4 * h + 3] += a.w;
          if (GLU) {
            if (p.split > 1) a = ld_cluster_f4(at + OUT * 4 + h * 16, s * CTAS + half);
            else a = *reinterpret_cast<const float4*>(smem + (row * SK_ROWS + OUT + g * 8) * 4 + h * 16);
            u[4 * h] += a.x; u[4 * h + 1] += a.y; u[4 * h + 2] += a.z; u[4 * h + 3] += a.w;
          }
        }
      }
      const float rs = p.row_scale != nullptr ? p.row_scale[t] : 1.f;
      float r[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int c = min(n + e, p.N - 1);
        if (GLU) {
          float x = v[e], y = u[e];
          if (FP8) {
            x *= rs;
            if (p.col_scale != nullptr) {
              x *= p.col_scale[c];
              y *= p.col_scale[p.up_row_offset + c];
            }
            r[e] = x / (1.f + __expf(-x)) * y * rs;
          } else if (p.acts.glu == GLU_GELU_TANH) {
            r[e] = epi_gelu_tanh(x) * y * rs;
          } else if (p.acts.glu == GLU_CLAMPED) {
            r[e] = epi_clamped(x * rs, y * rs, p.acts.limit, p.acts.alpha);
          } else {
            r[e] = x / (1.f + __expf(-x)) * y * rs;
          }
        } else {
          float x = v[e];
          if (FP8) {
            x *= p.col_scale != nullptr ? rs * p.col_scale[c] : rs;
            if (p.bias != nullptr) x += __bfloat162float(p.bias[c]);
          } else {
            if (p.bias != nullptr) x += __bfloat162float(p.bias[c]);
            if (p.acts.col_act != 0 && c >= p.acts.col_begin && c < p.acts.col_end) {
              const float z = fmaxf(x, 0.f);
              x = p.acts.col_act == COL_RELU2 ? z * z : epi_silu(x);
            }
            x *= rs;
          }
          r[e] = x;
        }
      }
      if (!GLU && p.logits != nullptr) {      // N is a multiple of 8 (checked by the launcher)
#pragma unroll
        for (int e = 0; e < 8; ++e) r[e] = __bfloat162float(__float2bfloat16_rn(r[e])) * p.logit_scale;
        float4* frow = reinterpret_cast<float4*>(p.logits + static_cast<long long>(t) * p.ldc + n);
        frow[0] = make_float4(r[0], r[1], r[2], r[3]);
        frow[1] = make_float4(r[4], r[5], r[6], r[7]);
        continue;
      }
      __nv_bfloat16* crow = p.C + static_cast<long long>(t) * p.ldc + n;
      if (n + 8 <= p.N) {
        *reinterpret_cast<uint4*>(crow) = make_uint4(pack_bf16x2(r[0], r[1]), pack_bf16x2(r[2], r[3]),
                                                     pack_bf16x2(r[4], r[5]), pack_bf16x2(r[6], r[7]));
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (n + e < p.N) crow[e] = __float2bfloat16_rn(r[e]);
      }
    }
    if (t1 < p.tn) __syncthreads();
  }
  if (CTAS * p.split > 1) {
    __syncwarp();
    cluster_sync_all();                     // the others may still read this CTA's part, or signal its barriers
  }
}

template <bool GLU, bool FP8, int KBS, bool PAIR>
static int launch_skinny(const CUtensorMap& tmA, const CUtensorMap& tmW, const SkinnyParams& p, int tiles, int smem,
                         cudaStream_t stream) {
  auto kern = gemm_skinny_kernel<GLU, FP8, KBS, PAIR>;
  static thread_local int configured_dev = -1;
  int dev = 0;
  cudaGetDevice(&dev);
  if (configured_dev != dev) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024);
    if (e != cudaSuccess) {
      set_last_error("cudaFuncSetAttribute(smem) failed: %s", cudaGetErrorString(e));
      return 1;
    }
    configured_dev = dev;
  }
  cudaLaunchConfig_t cfg = {};
  const int cluster = p.split * (PAIR ? 2 : 1);
  cfg.gridDim = dim3(tiles * cluster);
  cfg.blockDim = dim3(SK_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, tmA, tmW, p);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_last_error("gemm launch failed: %s", cudaGetErrorString(e));
    return 1;
  }
  return 0;
}

template <bool FP8, int KBS, bool PAIR>
static int launch_kind(const CUtensorMap& tmA, const CUtensorMap& tmW, const SkinnyParams& p, int glu, int tiles, int smem,
                       cudaStream_t stream) {
  return glu ? launch_skinny<true, FP8, KBS, PAIR>(tmA, tmW, p, tiles, smem, stream)
             : launch_skinny<false, FP8, KBS, PAIR>(tmA, tmW, p, tiles, smem, stream);
}

// Which products come here; the rest keeps the tiles of 128 or 256 rows of A. Measured on B200, weights from memory (us,
// tiles of A -> this kernel; the former also with elect.sync):
//   up to 80 rows: always. 4096x14336 62 -> 27 (48 rows), 8192x28672 124 -> 79, gated 2x14336x4096 67 -> 43, fp8 5120x25600
//     58 -> 34 (32 rows)
//   up to 160 rows: gated 2x28672x8192 184 -> 161 (100), 251 -> 171 (160). Not up to 128 rows where A is one tile of theirs and
//     the tiles of W are many waves here, each of which reads A again from L2: head 128256x4096 180 -> 187 (100) and 182 -> 192
//     (128), gated 2x25600x5120 94 -> 105 (128); but gated 2x14336x4096 52 -> 50 (128). Where K is not cut
//     (below), with few tiles only if it is long (fp8, 160 rows, 5120x25600 58 -> 49, but 6144x4096 15.7 -> 17.6)
//   up to 224 rows, as pairs, where the tiles fill the chip and are gated or long: gated 2x14336x4096 87 -> 58 (200),
//     2x28672x8192 217 -> 198, head 128256x8192 463 -> 438; but head 128256x4096 236 -> 238, and with 256 rows gated
//     2x25600x5120 128 -> 140
//   up to 256 rows where cutting K fills the chip and the parts are long enough to pay for adding 100 KB of sums:
//     8192x28672 107 -> 92 (200), 4096x14336 60 -> 39 (256); but 10240x8192 46 -> 55 (200), 6144x4096 22 -> 26 (256)
bool gemm_skinny_takes(bool fp8, bool cut, int M, int N, int K, bool glu) {
  if (M <= 80) return true;
  if (M > SK_MAX_TOKENS) return false;
  const int out = glu ? SK_ROWS / 2 : SK_ROWS;
  const int tiles = (N + out - 1) / out, sms = device_sm_count();
  const int num_kb = (K + (fp8 ? 127 : 63)) / (fp8 ? 128 : 64);
  if (!cut && M > 112 && tiles < sms && (M > 160 || num_kb < 128)) return false;
  if (M <= 160) return M > 128 || tiles <= (M <= 112 ? 4 : 2) * sms;
  if (M <= 224 && tiles >= sms && (glu || num_kb >= 128)) return true;
  return 2 * tiles <= sms && num_kb >= (M <= 208 ? 64 : 128);
}

// Pairs of CTAs read A once for 256 rows of W: from 113 rows on, where L2 would be read more for A than for W (160 rows, gated
// 2x28672x8192 177 -> 171 us, 5120x25600 61 -> 57, head 128256x8192 387 -> 376; 100 rows, 161 -> 162, 55 -> 54). With fewer tiles
// a cluster would be four pairs (4096x14336, 160 rows: 30 -> 48 us), and beyond 160 rows one CTA with all of K's sums is better.
static bool skinny_pairs(int M, int N, bool glu) {
  const int out = glu ? SK_ROWS / 2 : SK_ROWS;
  const int tiles = (N + out - 1) / out, sms = device_sm_count();
  return M > 112 && (M <= 160 ? 4 * tiles >= sms : tiles >= sms);
}

int gemm_skinny(bool fp8, bool cut, const void* A, long long lda, const void* W, long long ldw, long long rows_w, void* C,
                long long ldc, const void* bias, const float* row_scale, const float* col_scale, int M, int N, int K, int glu,
                int up_row_offset, const GemmActs& acts, uint32_t* status, cudaStream_t stream, float* logits,
                float logit_scale) {
  const int esz = fp8 ? 1 : 2, bk = fp8 ? 128 : 64;
  SkinnyParams p;
  const bool pair = skinny_pairs(M, N, glu != 0);
  const int ctas = pair ? 2 : 1;
  p.tn = pair ? (M + 31) / 32 * 32 : (M + 15) / 16 * 16;
  p.num_kb = (K + bk - 1) / bk;
  const int out = glu ? SK_ROWS / 2 : SK_ROWS;
  const int tiles = (N + ctas * out - 1) / (ctas * out), tile_ctas = tiles * ctas;
  const int sms = device_sm_count();
  const int kb_bytes = SK_W_BYTES + p.tn / ctas * 128;
  int dump = SK_ROWS * p.tn * 4;
  // Two CTAs per SM (one loads while the other starts or ends) where three stages of both fit: up to 160 rows.
  // Parts of K: doubled until the CTAs cover 0.6 of the SMs, half of them from 64 rows on, where the sums to be added weigh
  // more; more parts than that only add sums (48 rows, 6144x4096 in 2 / 4 parts: 14.8 / 16.2 us; 4096x4096 in 4 / 8: 12.1 /
  // 15.0; 128 rows, 5120x8192 in 2 / 4: 26.6 / 28.3). At least four k-blocks each, and never a second wave.
  // K stays whole where the caller wants it so, and for fp8: the sums of one accumulator over all of K are bit for bit those of
  // the tiles of A, and a last bit that differs moves the scale with which the next layer rounds a whole row to eight bits.
  const int two = 110 * 1024, one = 220 * 1024;
  const bool pairs = 3 * kb_bytes <= two;
  const int slots = pairs ? 2 * sms : sms;
  const int enough = sms * (M < 64 ? 6 : 5) / 10;
  int split = 1;
  while (cut && split * ctas * ctas < 8 && tile_ctas * split < enough && tile_ctas * split * 2 <= slots &&
         p.num_kb / (split * 2) >= 4 && (!pair || dump <= two)) split *= 2;
  p.split = split;
  // One CTA per SM sets the pace itself: two k-blocks per stage halve its waits, as long as four stages are left
  // (fp8 5120x25600, 1 row: 37 -> 30 us; 100 rows, three stages: 46 -> 55 us).
  const bool alone = !pairs || tile_ctas * split <= sms;
  const int kbs = !pair && alone && 8 * kb_bytes <= one ? 2 : 1;
  p.stages = min(SK_MAX_STAGES, (alone ? one : two) / (kbs * kb_bytes));
  p.dump_rows = p.tn;
  if (pair && split == 1 && dump > two) {
    p.dump_rows = 128;
    dump = SK_ROWS * 128 * 4;
  }
  int smem = p.stages * kbs * kb_bytes;
  if (smem < dump) smem = dump;
  if (smem < 80 * 1024) smem = 80 * 1024;   // at most two CTAs per SM: none waits for another's TMEM
  smem += 1024;
  p.tmem_cols = 32;
  while (p.tmem_cols < p.tn) p.tmem_cols *= 2;

  CUtensorMap tmA, tmW;
  {
    uint64_t dims[2] = {(uint64_t)K, (uint64_t)M};
    uint64_t strides[1] = {(uint64_t)lda * esz};
    uint32_t box[2] = {(uint32_t)bk, (uint32_t)(p.tn / ctas)};
    if (!(fp8 ? make_tensor_map_u8(&tmA, A, 2, dims, strides, box) : make_tensor_map_bf16(&tmA, A, 2, dims, strides, box)))
      return 1;
  }
  {
    uint64_t dims[2] = {(uint64_t)K, (uint64_t)rows_w};
    uint64_t strides[1] = {(uint64_t)ldw * esz};
    uint32_t box[2] = {(uint32_t)bk, (uint32_t)out};
    if (!(fp8 ? make_tensor_map_u8(&tmW, W, 2, dims, strides, box) : make_tensor_map_bf16(&tmW, W, 2, dims, strides, box)))
      return 1;
  }
  p.C = reinterpret_cast<__nv_bfloat16*>(C);
  p.logits = logits;
  p.logit_scale = logit_scale;
  p.ldc = ldc;
  p.bias = reinterpret_cast<const __nv_bfloat16*>(bias);
  p.row_scale = row_scale;
  p.col_scale = col_scale;
  p.M = M;
  p.N = N;
  p.up_row_offset = up_row_offset;
  p.acts = acts;
  p.status = status;
  if (pair)
    return fp8 ? launch_kind<true, 1, true>(tmA, tmW, p, glu, tiles, smem, stream)
               : launch_kind<false, 1, true>(tmA, tmW, p, glu, tiles, smem, stream);
  if (kbs == 2)
    return fp8 ? launch_kind<true, 2, false>(tmA, tmW, p, glu, tiles, smem, stream)
               : launch_kind<false, 2, false>(tmA, tmW, p, glu, tiles, smem, stream);
  return fp8 ? launch_kind<true, 1, false>(tmA, tmW, p, glu, tiles, smem, stream)
             : launch_kind<false, 1, false>(tmA, tmW, p, glu, tiles, smem, stream);
}

}  // namespace tw

using namespace tw;

// fp32 logits of a bf16 head, logits = scale * bf16(A W^T): what the product in bf16 and a conversion would give, without the trip
// through memory (200 rows of 128256x8192: 463 + 75 -> 438 us; 100 rows of 128256x4096: 180 + 33 -> 187, so here for every number
// of rows that fits).
extern "C" int tw_gemm_logits_takes(int M, int N, int K) {
  return M > 0 && M <= SK_MAX_TOKENS && N > 0 && N % 8 == 0 && K > 0 && K % 8 == 0;
}
extern "C" int tw_gemm_logits(const void* A, long long lda, const void* W, long long ldw, float* logits, long long ldc, float scale,
                              int M, int N, int K, uint32_t* status, cudaStream_t stream) {
  if (!tw_gemm_logits_takes(M, N, K) || lda % 8 != 0 || ldw % 8 != 0 || ldc % 4 != 0) {
    set_last_error("tw_gemm_logits: shape %d x %d x %d, strides %lld, %lld, %lld", M, N, K, lda, ldw, ldc);
    return 1;
  }
  return gemm_skinny(false, true, A, lda, W, ldw, N, nullptr, ldc, nullptr, nullptr, nullptr, M, N, K, 0, 0, GemmActs{}, status, stream,
                     logits, scale);
}
