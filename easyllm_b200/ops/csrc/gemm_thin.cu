// bf16 GEMM for few rows of activations (decoding, short prompts), sm_100a:  out[T, N] (+)= x[T, K] · W^T (+ bias).
//
// With few rows the product is bound by the bytes of W, and a grid of 128 x 256 output tiles leaves most SMs idle (16 tiles
// for N = 4096).  Here W is the M side of tcgen05.mma: a tile is 128 rows of W by BN rows of x (16 to 128), so 16 rows of x
// cost a sixteenth of a 256-wide tile, and the reduction is split over the CTAs of a cluster (1, 2, 4 or 8, picked by
// thin_split so that the tiles fill the SMs evenly).  The partial sums meet in shared memory: every CTA sends the fp32
// columns that a peer finishes to that peer (distributed shared memory, an mbarrier per direction), and each sums its
// columns in the order of the cluster's ranks, so results do not depend on timing and no workspace exists.
//   warp 0     TMA producer: a [128 x 64] box of W and a [BN x 64] box of x per stage
//   warp 1     issues tcgen05.mma (128 x BN x 16); two accumulators in TMEM
//   warps 2-5  TMEM -> peers' shared memory -> sum -> bias -> global; a warp stores 32 consecutive columns of a row
// W_MN: W is stored [K, N] (the input gradient of a linear layer reads its weight in place).
#include "gemm_fuse.cuh"

namespace ell {

constexpr int kThRows = 128;               // rows of W of a tile
constexpr int kThWBytes = kThRows * kBK * 2;
constexpr int kThAhead = 16;               // k-blocks of W fetched into L2 ahead of the wait: 39 MB over the SMs

template <int BN>
struct ThinCfg {
  static constexpr int kStageBytes = kThWBytes + BN * kBK * 2;
  static constexpr int kStages = BN >= 128 ? 4 : (BN >= 64 ? 6 : 8);
  static constexpr int kExCols = BN < 64 ? BN : 64;        // columns of an exchange between CTAs
  static constexpr int kExBytes = kThRows * kExCols * 4;   // of each direction
  static constexpr int kTmemCols = 2 * BN < 32 ? 32 : 2 * BN;
  static constexpr int kSmemBytes = kStages * kStageBytes + 2 * kExBytes + 1024 + 256;
};

struct ThinShared {
  uint64_t full[8], empty[8], tmem_full[2], tmem_empty[2], recv_full, recv_free;
  uint32_t tmem_base;
  int abort_flag;
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_to_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// Shared memory of this CTA -> shared memory of a peer, whose mbarrier counts the bytes.
__device__ __forceinline__ void bulk_copy_to_peer(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "r"(smem_u32(src)), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
// As mbar_wait, for a barrier that other CTAs of the cluster arrive on.
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                                  unsigned long long limit_ns) {
  const unsigned long long t0 = globaltimer_ns();
  uint32_t spins = 0;
  while (true) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    if (ok) return true;
    if ((++spins & 255u) == 0 && (*abort_flag || globaltimer_ns() - t0 > limit_ns)) return false;
  }
}

__device__ __forceinline__ void set_in_peer(uint32_t addr, int v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
// The whole cluster stops waiting: a CTA that gave up may still be sent to, and its copies may still be on their way.
__device__ __forceinline__ void give_up(ThinShared* sh, int split) {
  sh->abort_flag = 1;
  for (int r = 0; r < split && split > 1; ++r) set_in_peer(map_to_rank(smem_u32(&sh->abort_flag), r), 1);
}

// Barrier of the epilogue that tells every thread whether any of them failed.
__device__ __forceinline__ bool epi_any(bool failed) {
  uint32_t any;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
      "bar.red.or.pred p, 1, %2, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(any) : "r"((uint32_t)failed), "n"(kEpiThreads) : "memory");
  return any != 0;
}

// Rows of x of a tile.
__host__ __device__ __forceinline__ int thin_bn(int T) { return T <= 16 ? 16 : (T <= 32 ? 32 : (T <= 64 ? 64 : 128)); }

struct ThinArgs {
  void* out;
  const __nv_bfloat16* bias;
  int T, N, K, ldo, out_mode, split, split_log2;
  unsigned long long limit_ns;   // of a wait for a peer
  int mute;                      // CTA of a cluster that sends nothing (a test of the waits), or -1
  int* err;
};

// k-blocks [first, last) of CTA r out of `split`
__host__ __device__ __forceinline__ int thin_first_block(int blocks, int split, int r) { return (int)((long long)blocks * r / split); }

// Sums of `cols` columns over the CTAs of the cluster, in the order of their ranks; CH columns at a time so that their loads
// are in flight together.
template <int CH, typename Old, typename Put>
__device__ __forceinline__ void sum_columns(const float* mine, const float* theirs, int cols, int rank, int split, int t, int T,
                                            const Old& old, const Put& put) {
#pragma unroll 1
  for (int j = 0; j < cols && t + j < T; j += CH) {
    float s[CH], before[CH];
#pragma unroll
    for (int i = 0; i < CH; ++i) {
      s[i] = 0.f;
      before[i] = t + j + i < T ? old(t + j + i) : 0.f;
    }
#pragma unroll 1
    for (int p = 0; p < split; ++p) {
      const float* src = (p == rank ? mine : theirs + (size_t)(p - (p > rank)) * cols * kThRows) + j * kThRows;
#pragma unroll
      for (int i = 0; i < CH; ++i) s[i] += src[i * kThRows];
    }
#pragma unroll
    for (int i = 0; i < CH; ++i)
      if (t + j + i < T) put(t + j + i, before[i] + s[i]);
  }
}

template <int BN, bool W_MN>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_thin_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const ThinArgs a) {
  using Cfg = ThinCfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  // the same offset in every CTA of the cluster: the dynamic shared memory starts at the same address in each
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sW = smem;
  uint8_t* sX = smem + Cfg::kStages * kThWBytes;
  float* send = reinterpret_cast<float*>(smem + Cfg::kStages * Cfg::kStageBytes);   // [column][row]
  float* recv = send + Cfg::kExBytes / 4;                                            // [peer][column][row]
  ThinShared* sh = reinterpret_cast<ThinShared*>(recv + Cfg::kExBytes / 4);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int split = a.split, rank = split > 1 ? (int)cluster_rank() : 0;
  const int tiles_t = (a.T + BN - 1) / BN, tiles = tiles_t * ((a.N + kThRows - 1) / kThRows);
  const int blocks = (a.K + kBK - 1) / kBK;
  const int kb0 = thin_first_block(blocks, split, rank), kb1 = thin_first_block(blocks, split, rank + 1);
  const int first = blockIdx.x / split, step = gridDim.x / split;

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::kStages; ++s) {
      mbar_init(&sh->full[s], 1);
      mbar_init(&sh->empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&sh->tmem_full[i], 1);
      mbar_init(&sh->tmem_empty[i], kEpiThreads);
    }
    mbar_init(&sh->recv_full, 1);                    // and the peers' bytes
    mbar_init(&sh->recv_free, 4 * (split - 1) + (split == 1));   // one arrival per epilogue warp of a peer
    sh->abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  if (warp == 1) tmem_alloc<Cfg::kTmemCols>(&sh->tmem_base);
  tc_fence_before();
  __syncthreads();
  if (split > 1) cluster_sync_all();                 // the peers' barriers exist
  tc_fence_after();
  const uint32_t tmem_base = sh->tmem_base;
  volatile int* abort_flag = &sh->abort_flag;
  chain_next();
  if (threadIdx.x == 0 && first < tiles) {
    // the weight's first blocks come into L2 while the kernel before this one ends
    const int n0 = first / tiles_t * kThRows;
    for (int kb = kb0; kb < min(kb1, kb0 + kThAhead); ++kb) {
      if (!W_MN) {
        tma_prefetch_l2_2d(&tmW, kb * kBK, n0);
      } else {
        tma_prefetch_l2_2d(&tmW, n0, kb * kBK);
        tma_prefetch_l2_2d(&tmW, n0 + 64, kb * kBK);
      }
    }
  }
  chain_wait();

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = first; tile < tiles && ok; tile += step) {
        const int n0 = tile / tiles_t * kThRows, t0 = tile % tiles_t * BN;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&sh->empty[stage], phase ^ 1, abort_flag)) {
            ok = false;
            break;
          }
          mbar_expect_tx(&sh->full[stage], Cfg::kStageBytes);
          uint8_t* w = sW + stage * kThWBytes;
          if (!W_MN) {
            tma_load_2d(w, &tmW, &sh->full[stage], kb * kBK, n0);
          } else {
            tma_load_2d(w, &tmW, &sh->full[stage], n0, kb * kBK);
            tma_load_2d(w + 64 * kBK * 2, &tmW, &sh->full[stage], n0 + 64, kb * kBK);
          }
          tma_load_2d(sX + stage * (BN * kBK * 2), &tmX, &sh->full[stage], kb * kBK, t0);
          if (++stage == Cfg::kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      if (!ok) {
        give_up(sh, split);
        atomicCAS(a.err, 0, kErrProducer);
      }
    }
  } else if (warp == 1) {
    {                                                // the whole warp, see sm100.cuh
      const uint32_t e = elect_one(), tm = __reduce_or_sync(0xffffffffu, tmem_base);
      constexpr uint32_t idesc = make_idesc_bf16(kThRows, BN, W_MN, false);
      constexpr uint32_t w_lbo = W_MN ? 64 * kBK * 2 : 16, w_kstep = W_MN ? 2048 : 32;
      const uint64_t w_desc = make_smem_desc(smem_u32(sW), w_lbo, 1024), x_desc = make_smem_desc(smem_u32(sX), 16, 1024);
      int stage = 0, it = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = first; warp_uniform(tile < tiles) && ok; tile += step, ++it) {
        const int acc = it & 1;
        if (!mbar_wait_warp(&sh->tmem_empty[acc], ((it >> 1) & 1) ^ 1, abort_flag)) {
          ok = false;
          break;
        }
        tc_fence_after();
        for (int kb = kb0; warp_uniform(kb < kb1); ++kb) {
          if (!mbar_wait_warp(&sh->full[stage], phase, abort_flag)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint64_t dw = w_desc + stage * (kThWBytes >> 4), dx = x_desc + stage * ((BN * kBK * 2) >> 4);
          const uint32_t add = warp_uniform(kb > kb0);
#pragma unroll
          for (int k = 0; k < kBK / 16; ++k)
            umma_bf16_warp(e, tm + acc * BN, dw + ((k * w_kstep) >> 4), dx + ((k * 32) >> 4), idesc, add | k);
          umma_commit_warp(e, &sh->empty[stage]);
          if (++stage == Cfg::kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (ok) umma_commit_warp(e, &sh->tmem_full[acc]);
      }
      if (!ok && e) {
        give_up(sh, split);
        atomicCAS(a.err, 0, kErrMma);
      }
    }
  } else {
    const int q = warp & 3, row = q * 32 + lane;     // TMEM lane = row of W in the tile
    constexpr int EX = Cfg::kExCols;
    const int cols = EX >> a.split_log2;             // columns (rows of x) of an exchange this CTA finishes
    const uint32_t block = (uint32_t)cols * kThRows * 4;
    int it = 0, ex = 0;
    bool failed = false;
    // A wait that runs out is one thread's own finding.  It stays set until the next vote, where all threads of the epilogue leave
    // together: one that left alone would strand the others at their barrier.
    for (int tile = first; tile < tiles; tile += step, ++it) {
      const int n0 = tile / tiles_t * kThRows, t0 = tile % tiles_t * BN, n = n0 + row;
      const int acc = it & 1;
      failed = epi_any(failed || !mbar_wait(&sh->tmem_full[acc], (it >> 1) & 1, abort_flag));
      if (failed) break;
      tc_fence_after();
      const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + acc * BN;
      const float bias = a.bias != nullptr && n < a.N ? __bfloat162float(a.bias[n]) : 0.f;
      auto put = [&](int t, float v) {
        const size_t at = (size_t)t * a.ldo + n;
        if (a.out_mode == kOutBf16) reinterpret_cast<__nv_bfloat16*>(a.out)[at] = __float2bfloat16_rn(v + bias);
        else reinterpret_cast<float*>(a.out)[at] = v;
      };
      auto old = [&](int t) {
        return a.out_mode == kOutF32Accum ? reinterpret_cast<const float*>(a.out)[(size_t)t * a.ldo + n] : 0.f;
      };
      if (split == 1) {
#pragma unroll 1
        for (int c = 0; c < BN && t0 + c < a.T; c += 16) {
          uint32_t v[16];
          tmem_ld_32x16(t_row + c, v);
          tmem_ld_wait();
          if (n < a.N) {
            float before[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) before[i] = t0 + c + i < a.T ? old(t0 + c + i) : 0.f;
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (t0 + c + i < a.T) put(t0 + c + i, before[i] + __uint_as_float(v[i]));
          }
          __syncwarp();                              // lanes past N skip the stores; the next load takes the whole warp
        }
        tc_fence_before();
        mbar_arrive(&sh->tmem_empty[acc]);
        continue;
      }
      for (int c0 = 0; c0 < BN; c0 += EX, ++ex) {
        // the peers are done with the exchange before: its bytes have left `send`, and their `recv` may be written
        if (ex > 0 && !mbar_wait_cluster(&sh->recv_free, (ex - 1) & 1, abort_flag, a.limit_ns)) failed = true;
#pragma unroll 1
        for (int c = 0; c < EX; c += 16) {
          uint32_t v[16];
          tmem_ld_32x16(t_row + c0 + c, v);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) send[(c + i) * kThRows + row] = __uint_as_float(v[i]);
        }
        if (c0 + EX == BN) {
          tc_fence_before();
          mbar_arrive(&sh->tmem_empty[acc]);
        }
        fence_proxy_async_smem();
        failed = epi_any(failed);
        if (failed) break;
        if (threadIdx.x == 64) {
          mbar_expect_tx(&sh->recv_full, (split - 1) * block);
          for (int d = 1; d < split && rank != a.mute; ++d) {          // slot of this CTA at peer p: its rank among the others
            const int p = (rank + d) & (split - 1);
            bulk_copy_to_peer(map_to_rank(smem_u32(recv), p) + (rank - (rank > p)) * block, send + (size_t)p * cols * kThRows,
                              block, map_to_rank(smem_u32(&sh->recv_full), p));
          }
        }
        if (!mbar_wait_cluster(&sh->recv_full, ex & 1, abort_flag, a.limit_ns)) {
          failed = true;
          give_up(sh, split);
        } else if (n < a.N) {
          const int tc = t0 + c0 + rank * cols;
          const float *mine = send + (size_t)rank * cols * kThRows + row, *theirs = recv + row;
          if (cols >= 8) sum_columns<8>(mine, theirs, cols, rank, split, tc, a.T, old, put);
          else if (cols == 4) sum_columns<4>(mine, theirs, cols, rank, split, tc, a.T, old, put);
          else sum_columns<2>(mine, theirs, cols, rank, split, tc, a.T, old, put);
        }
        fence_proxy_async_smem();                    // these reads before the peers' next copies
        __syncwarp();
        if (lane < split && lane != rank) mbar_arrive_cluster(map_to_rank(smem_u32(&sh->recv_free), lane));
      }
    }
    if (failed) {
      give_up(sh, split);
      atomicCAS(a.err, 0, kErrEpilogue);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (split > 1) cluster_sync_all();                 // no CTA starts a copy any more
  if (*abort_flag) {                                 // the same in the whole CTA behind either barrier
    // error path: give copies and MMAs in flight time to land before shared memory and TMEM go away
    const unsigned long long t0 = globaltimer_ns();
    while (threadIdx.x == 0 && globaltimer_ns() - t0 < 200000ull) {
    }
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc<Cfg::kTmemCols>(tmem_base);
  }
}

int make_tmap_bf16_2d(CUtensorMap* map, const void* ptr, uint64_t inner, uint64_t outer, uint64_t row_stride_bytes,
                      uint32_t box_inner, uint32_t box_outer);

// Estimated time of a launch with `s` CTAs per reduction, in us.  From trains of launches on weights that L2 does not hold:
// a launch costs 4.5; a k-block 0.27 plus what its rows of x add, 0.05 more with the traffic of more CTAs; a tile's end 0.3,
// or 1.2 with the exchange, plus the columns it writes, half of it hidden behind the next tile's loads.  Within 10 % of what was measured for N 1024 .. 11264, K 1024 .. 11008.
static float thin_us(int T, int N, int K, int s, int clusters) {
  const int bn = thin_bn(T), tiles = (T + bn - 1) / bn * ((N + kThRows - 1) / kThRows), blocks = (K + kBK - 1) / kBK;
  const int rounds = (tiles + clusters - 1) / clusters, own = (blocks + s - 1) / s;
  const float end = s > 1 ? 1.2f + 0.03f * bn : 0.3f + 0.01f * bn;
  const float us = 4.5f + rounds * own * (0.27f + 0.0004f * bn + (s > 1 ? 0.05f : 0.f)) + end * (rounds + 1) / 2;
  return fmaxf(us, 4.5f + (float)N * K * 2 / 6e6f);
}

static int thin_split(int T, int N, int K, const int* clusters, float* us) {
  int best = 1;
  *us = 1e30f;
  for (int i = 0, s = 1; i < 4 && s <= (K + kBK - 1) / kBK && clusters[i] > 0; s *= 2, ++i) {
    const float t = thin_us(T, N, K, s, clusters[i]);
    if (t < *us) {
      *us = t;
      best = s;
    }
  }
  return best;
}

template <int BN, bool W_MN>
static int launch_thin(const CUtensorMap& tw, const CUtensorMap& tx, ThinArgs a, cudaStream_t stream) {
  auto kern = gemm_thin_kernel<BN, W_MN>;
  cudaLaunchConfig_t cfg{};
  cfg.blockDim = dim3(kGemmThreads);
  cfg.dynamicSmemBytes = ThinCfg<BN>::kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute at[2] = {};
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  // clusters of 1, 2, 4, 8 CTAs that are resident together: a cluster lies within one GPC, so fewer than SMs / size
  static int clusters[4] = {0, 0, 0, 0};
  if (clusters[0] == 0) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, ThinCfg<BN>::kSmemBytes);
    if (e != cudaSuccess) return (int)e;
    int found[4] = {0, 0, 0, 0}, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&found[0], cudaDevAttrMultiProcessorCount, dev);
    for (int i = 1; i < 4; ++i) {
      at[0].val.clusterDim.x = 1 << i;
      cfg.gridDim = dim3(1 << i);
      cfg.numAttrs = 1;
      if (cudaOccupancyMaxActiveClusters(&found[i], kern, &cfg) != cudaSuccess) {
        cudaGetLastError();
        found[i] = 0;
      }
    }
    for (int i = 3; i >= 0; --i) clusters[i] = found[i];
  }
  const int tiles = (a.T + BN - 1) / BN * ((a.N + kThRows - 1) / kThRows);
  float us;
  if (a.split == 0) a.split = thin_split(a.T, a.N, a.K, clusters, &us);
  a.split_log2 = __builtin_ctz(a.split);
  const int fit = clusters[a.split_log2];
  if (fit < 1) return -2;
  cfg.gridDim = dim3((tiles < fit ? tiles : fit) * a.split);
  at[0].val.clusterDim.x = a.split;
  cfg.numAttrs = 2;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, tw, tx, a);
  return e != cudaSuccess ? (int)e : launch_status();
}

}  // namespace ell

using namespace ell;

// The kernel for a product of T rows with an N x K weight: 0 the 128 x 256 tiles (or CTA pairs), 1 this file's, 2 the
// matrix-vector kernel (16 rows and fewer).  Estimates in us, fitted to the same trains of launches as thin_us:
//   tiles        4 + 0.39 a k-block and round of 148 tiles, at least 4 + the weight at 5.3 TB/s
//   matrix-vector  3 + 2.6 per 1024 of K (its warps split K no further than 8 ways), at least 3 + the weight at 4.7 TB/s, 3.6
//                with more than 8 rows; with so few columns that its CTAs do not fill the GPU it is the launch alone
// E.g. 1 row, 4096 x 11008: 20.7 here, 34 matrix-vector, 68 tiles; 2048 x 1024: 6.7, 4.9, 10.8; 64 rows of 22016 x 4096: 41.8
// here, 38.7 tiles.
ELL_API int ell_gemm_thin_route(int T, int N, int K) {
  // clusters of 1, 2, 4, 8 CTAs that fit on a B200
  static const int clusters[4] = {148, 74, 36, 16};
  if (T <= 0 || N <= 0 || K <= 0 || T > 256) return 0;
  float thin;
  thin_split(T, N, K, clusters, &thin);
  const float bytes = (float)N * K * 2;
  const int tiles = (T + 127) / 128 * ((N + 255) / 256), rounds = (tiles + kNumSMs - 1) / kNumSMs;
  const float tiled = fmaxf(4.f + 0.39f * rounds * ((K + kBK - 1) / kBK), 4.f + bytes / 5.3e6f);
  if (T <= 16) {
    const float mv = N < 512 ? 3.f : fmaxf(3.f + 2.6e-3f * K, 3.f + bytes / (T <= 8 ? 4.7e6f : 3.6e6f));
    if (mv <= thin && mv <= tiled) return 2;
  }
  return thin < tiled ? 1 : 0;
}

// out [T, N] rows of ldo = x [T, K] rows of ldx · W^T (+ bias [N], bf16 output only); W [N, K] (w_mn 0) or [K, N] (w_mn 1),
// rows of ldw.  out_mode: 0 bf16, 1 fp32 +=, 2 fp32 =.  K, ldx, ldw multiples of 8, x and W on 16-byte boundaries.
// split: CTAs per reduction, 0 for the rule above.  wait_us: limit of the wait for another CTA's sums (0: 2 s), after which the error
// word is set; mute: CTA of a cluster that withholds its sums, so that a test can let that wait run out (-1: none).
ELL_API int ell_gemm_thin(const void* x, const void* W, void* out, const void* bias, int T, int N, int K, int ldx, int ldw,
                          int ldo, int w_mn, int out_mode, int split, int wait_us, int mute, int* err, cudaStream_t stream) {
  if (T <= 0 || N <= 0 || K <= 0) return 0;
  if (out_mode < kOutBf16 || out_mode > kOutF32 || (bias && out_mode != kOutBf16)) return -2;
  if (split != 0 && split != 1 && split != 2 && split != 4 && split != 8) return -2;
  const int BN = thin_bn(T);
  CUtensorMap tw, tx;
  int rc = w_mn ? make_tmap_bf16_2d(&tw, W, (uint64_t)N, (uint64_t)K, (uint64_t)ldw * 2, 64, kBK)
                : make_tmap_bf16_2d(&tw, W, (uint64_t)K, (uint64_t)N, (uint64_t)ldw * 2, kBK, kThRows);
  if (!rc) rc = make_tmap_bf16_2d(&tx, x, (uint64_t)K, (uint64_t)T, (uint64_t)ldx * 2, kBK, BN);
  if (rc) return rc;
  if (split > (K + kBK - 1) / kBK) return -2;
  const unsigned long long limit = wait_us > 0 ? wait_us * 1000ull : kWaitTimeoutNs;
  const ThinArgs a{out, (const __nv_bfloat16*)bias, T, N, K, ldo, out_mode, split, 0, limit, mute, err};
#define ELL_THIN(BN_)                                                                     \
  if (BN == BN_) return w_mn ? launch_thin<BN_, true>(tw, tx, a, stream) : launch_thin<BN_, false>(tw, tx, a, stream);
  ELL_THIN(16)
  ELL_THIN(32)
  ELL_THIN(64)
  ELL_THIN(128)
#undef ELL_THIN
  return -3;
}
