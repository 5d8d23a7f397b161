// Causal flash attention backward on tcgen05 / TMEM for sm_100a: packed variable-length documents,
// MHA and GQA, head_dim 128, bf16 in/out, fp32 accumulation.
//
// Two kernels, one for the keys and one for the queries; both compute the scores and dP:
//   S  = Q K^T       P  = exp2(S*scale*log2e - lse*log2e)        (causal / document mask)
//   dP = dO V^T      dS = P * (dP - delta) * scale               delta = rowsum(dO * O)
//   dV += P^T dO     dK += dS^T Q                                dQ += dS K
// That is seven products where one kernel for all needs five, but nothing leaves a CTA before it is finished.  The one kernel walked
// the queries of a key tile and added every dQ tile to fp32 memory: S, P, dP, dS, dQ and the drain of dQ were a chain of 6500 cycles a
// step (five products take 2560), 64 KB of fp32 went through shared memory twice a step, and dQ came out in the order the CTAs
// ended.  Here P, dP and dS stay in TMEM, as operands of the products with them, and the chain of a step is the softmax threads' own work.
//
// 640 threads:
//   warp 0      TMA loads
//   warp 1      issues the products (the whole warp walks the loop, see sm100.cuh)
//   warp 2      statistics of the query tile (keys kernel) / work items (queries kernel)
//   warps 4-19  four groups of 128 threads; a thread owns one TMEM lane and a quarter of the 128 columns, and turns S into P and dP
//               into dS.  (Two groups with 64 columns a thread have half the warps to hide the chain's latencies: keys kernel 271 us
//               where four take 258, queries kernel 220 and 217; 4096 tokens, 32 heads.)
// Keys kernel: one CTA per (128-key tile, kv head); lanes are keys, columns queries.  TMEM: S | P^T 0-127, dP | dS^T 128-255, dV 256-383,
//   dK 384-511.  dV(i) and S(i+1) run while dS(i) is made, dK(i) and dP(i+1) while P(i+1) is: a step is as long as its P and dS passes.
// Queries kernel: CTAs take (128-query tile, head) items as they get free; lanes are queries, columns keys.  TMEM: S 0-127, dP | dS of
//   even steps 128-255, of odd steps 256-383, dQ 384-511.
// What bounds them: of 3250 cycles a step in the keys kernel 1550 are the P pass (1024 of them the special-function unit's), 750 the dS
// pass, the rest hand-overs and TMEM loads; products take 2048.  us, one B200, inputs not in L2, row sums included, before -> now: 4096
// tokens, 32 heads 587 -> 482; 8 documents of 512, 32 heads on 8 216 -> 171; 3001 tokens in 7 documents, 16 on 4 114 -> 99; 200 tokens,
// 8 heads 38 -> 30.  Exponentials of a quarter of the columns on the FMA pipe: keys kernel 250 us, queries kernel 221; not worth
// their error of 7e-5.
// dS and P^T of a thread's columns go over its own columns of dP and S only: those of another group may not have been read yet.
// The transposed operands (dO, Q, K as [k x n]) are read in place with MN-major descriptors, so nothing is transposed in memory.
// Every wait is bounded; on expiry the CTA records an error code, lets go of everything, frees its TMEM and returns.
//
// Backward of flash_attn_varlen_{qkv,kv}packed_func used by the reference
// (llm/models/mg_models/llama/transformer.py:65-143).
#include "common.cuh"
#include "sm100.cuh"

namespace ell {
using namespace sm100;

constexpr int kFbThreads = 640, kFbSoftmaxWarps = 16;
constexpr int kFbRegsIo = 64, kFbRegsSoftmax = 104;    // of the launch's 96 x 640
constexpr int kFbTile = 128, kFbD = 128;
constexpr int kFbTileBytes = 128 * 128 * 2;   // 32 KiB
constexpr int kFbHalf = kFbTileBytes / 2;     // 16 KiB: one 64-column half of a tile

enum FbErr { kFbErrProducer = 21, kFbErrMma = 22, kFbErrSoftmax = 23, kFbErrStats = 24 };

struct FbArgs {
  const float *lse, *delta;             // [Hq, T]
  const int* row_start;
  int T, Hq, Hk, nsplit;                // nsplit: CTAs that share the query heads of a kv head (keys kernel)
  float scale;
  const float* alibi_slopes;
  int* err;
};

// Index one past the last query tile that can see keys up to k_last: row_start is non-decreasing, so the
// tiles whose first row starts a document after k_last (and all later tiles) are invisible.  Warp-uniform.
__device__ __forceinline__ int fb_last_qtile(const int* __restrict__ row_start, int j, int n_qt, int k_last, int lane) {
  int i_end = j + 1;
  for (int base = j + 1; base < n_qt; base += 32) {
    const int i = base + lane;
    const bool vis = i < n_qt && row_start[i * kFbTile] <= k_last;
    const unsigned m = __ballot_sync(0xffffffffu, vis);
    i_end = base + __popc(m);
    if (m != 0xffffffffu) break;
  }
  return i_end;
}

__device__ __forceinline__ void fb_load_tile(uint8_t* dst, const CUtensorMap* map, uint64_t* bar, int x, int row) {
  tma_load_2d(dst, map, bar, x, row);
  tma_load_2d(dst + kFbHalf, map, bar, x + 64, row);
}

__device__ __forceinline__ uint32_t fb_pack(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// Bits [lo, hi] of 32, both ends clipped.
__device__ __forceinline__ uint32_t fb_bits(int lo, int hi) {
  if (hi < 0 || lo > 31) return 0u;
  const uint32_t m = 0xffffffffu >> (31 - min(hi, 31));
  return lo > 0 ? m & (0xffffffffu << lo) : m;
}

// Of 32 raw scores those whose bit in `seen` is clear become -inf, so that their exponential is 0.
__device__ __forceinline__ void fb_mask32(uint32_t* v, uint32_t seen) {
  if (__any_sync(0xffffffffu, seen != 0xffffffffu)) {
#pragma unroll
    for (int e = 0; e < 32; ++e)
      if (!(seen >> e & 1)) v[e] = 0xff800000u;
  }
}

// dS = P * (dP - delta) * scale for 32 columns, two at a time: (dP * scale - delta * scale), then times P.
// p: 16 packed pairs; nd: -delta * scale of a column pair.
template <typename Nd>
__device__ __forceinline__ void fb_ds32(const uint32_t* v, const uint32_t* p, float scale, Nd nd, uint32_t* out) {
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    const float2 pp = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&p[e]));
    const float2 t = ffma2(make_float2(__uint_as_float(v[2 * e]), __uint_as_float(v[2 * e + 1])), make_float2(scale, scale), nd(e));
    const float2 ds = ffma2(pp, t, make_float2(0.f, 0.f));
    out[e] = fb_pack(ds.x, ds.y);
  }
}

// 64 fp32 columns of this warp's TMEM lanes -> bf16 [32 rows x 64 columns] in shared memory, in the 128-byte swizzle of a TMA store.
__device__ __forceinline__ void fb_stage64(uint32_t t_src, uint8_t* stage, int lane) {
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    uint32_t v[32];
    tmem_ld_32x32(t_src + c * 32, v);
    tmem_ld_wait();
#pragma unroll
    for (int g8 = 0; g8 < 4; ++g8)
      *reinterpret_cast<uint4*>(stage + lane * 128 + (((c * 4 + g8) ^ (lane & 7)) << 4)) =
          make_uint4(fb_pack(__uint_as_float(v[g8 * 8]), __uint_as_float(v[g8 * 8 + 1])),
                     fb_pack(__uint_as_float(v[g8 * 8 + 2]), __uint_as_float(v[g8 * 8 + 3])),
                     fb_pack(__uint_as_float(v[g8 * 8 + 4]), __uint_as_float(v[g8 * 8 + 5])),
                     fb_pack(__uint_as_float(v[g8 * 8 + 6]), __uint_as_float(v[g8 * 8 + 7])));
  }
  fence_proxy_async_smem();
  __syncwarp();
}

// ------------------------------------------------ keys ------------------------------------------------
struct FbKvShared {
  uint64_t kv_full, q_full[2], q_empty[2], do_full[2], do_empty[2], st_full[2], st_empty[2], s_full, dp_full, p_full, ds_full, done;
  float lse2[2][kFbTile], nds[2][kFbTile];     // -lse * log2(e), -delta * scale
  int start[2][kFbTile];
  uint32_t tmem_base;
  int abort_flag;
};
constexpr int kFbKvSmem = 6 * kFbTileBytes + 1024 + 4096;   // K, V, Q x2, dO x2
static_assert(sizeof(FbKvShared) <= 4096, "");

__global__ void __launch_bounds__(kFbThreads, 1)
flash_bwd_kv_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                    const __grid_constant__ CUtensorMap tmdK, const __grid_constant__ CUtensorMap tmdV,
                    const __grid_constant__ FbArgs fa) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t *sK = smem, *sV = smem + kFbTileBytes, *sQ = smem + 2 * kFbTileBytes, *sdO = smem + 4 * kFbTileBytes;
  FbKvShared* sh = reinterpret_cast<FbKvShared*>(smem + 6 * kFbTileBytes);
  int* const err = fa.err;
  const int T = fa.T;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int n_qt = (T + kFbTile - 1) / kFbTile;
  // blockIdx.y = key tile (j = 0 has the longest walk; with x varying fastest the heaviest CTAs of every head
  // are scheduled first), blockIdx.x = kv head x split of its query-head group.
  const int j = blockIdx.y;
  const int kvh = blockIdx.x / fa.nsplit;
  const int G = fa.Hq / fa.Hk / fa.nsplit;     // query heads walked by this CTA
  const int h_first = kvh * (fa.Hq / fa.Hk) + (blockIdx.x % fa.nsplit) * G;
  const int k0 = j * kFbTile;
  const int k_last = min(k0 + kFbTile, T) - 1;

  if (threadIdx.x == 0) {
    mbar_init(&sh->kv_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&sh->q_full[s], 1);
      mbar_init(&sh->q_empty[s], 1);
      mbar_init(&sh->do_full[s], 1);
      mbar_init(&sh->do_empty[s], 1);
      mbar_init(&sh->st_full[s], 1);
      mbar_init(&sh->st_empty[s], kFbSoftmaxWarps);
    }
    mbar_init(&sh->s_full, 1);
    mbar_init(&sh->dp_full, 1);
    mbar_init(&sh->p_full, kFbSoftmaxWarps);
    mbar_init(&sh->ds_full, kFbSoftmaxWarps);
    mbar_init(&sh->done, 1);
    sh->abort_flag = *(volatile int*)err;      // an earlier CTA already failed: do not wait on anything
    fence_barrier_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmdO);
  }
  if (warp == 1) tmem_alloc<512>(&sh->tmem_base);
  const int i_end = fb_last_qtile(fa.row_start, j, n_qt, k_last, lane);
  const int n_q = i_end - j, n_it = G * n_q;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = sh->tmem_base;
  const bool dead_on_arrival = sh->abort_flag != 0;
  volatile int* abort_flag = &sh->abort_flag;

  if (dead_on_arrival) {
    // fall through to the common exit: nothing was issued
  } else if (warp < 4) {
    setmaxnreg_dec<kFbRegsIo>();
    if (warp == 0 && lane == 0) {
      // ------------------------------- TMA loads -------------------------------
      bool ok = true;
      mbar_expect_tx(&sh->kv_full, 2 * kFbTileBytes);
      fb_load_tile(sK, &tmK, &sh->kv_full, kvh * kFbD, k0);
      fb_load_tile(sV, &tmV, &sh->kv_full, kvh * kFbD, k0);
      int it = 0;
      for (int g = 0; g < G && ok; ++g) {
        const int x = (h_first + g) * kFbD;
        for (int i = j; i < i_end; ++i, ++it) {
          const int s = it & 1;
          const uint32_t ph = ((it >> 1) & 1) ^ 1;
          if (!mbar_wait(&sh->q_empty[s], ph, abort_flag)) { ok = false; break; }
          mbar_expect_tx(&sh->q_full[s], kFbTileBytes);
          fb_load_tile(sQ + s * kFbTileBytes, &tmQ, &sh->q_full[s], x, i * kFbTile);
          if (!mbar_wait(&sh->do_empty[s], ph, abort_flag)) { ok = false; break; }
          mbar_expect_tx(&sh->do_full[s], kFbTileBytes);
          fb_load_tile(sdO + s * kFbTileBytes, &tmdO, &sh->do_full[s], x, i * kFbTile);
        }
      }
      if (!ok) {
        sh->abort_flag = 1;
        atomicCAS(err, 0, kFbErrProducer);
      }
    } else if (warp == 1) {
      // ------------------------------- MMA issuer -------------------------------
      constexpr uint32_t idesc_kk = make_idesc_bf16(128, 128, false, false);  // A, B K-major
      constexpr uint32_t idesc_km = make_idesc_bf16(128, 128, false, true);   // A K-major (TMEM), B MN-major
      const uint32_t e = elect_one(), tm = __reduce_or_sync(0xffffffffu, tmem_base);
      const uint64_t k_kk = make_smem_desc(smem_u32(sK), 16, 1024), v_kk = make_smem_desc(smem_u32(sV), 16, 1024);
      const uint64_t q_kk = make_smem_desc(smem_u32(sQ), 16, 1024), do_kk = make_smem_desc(smem_u32(sdO), 16, 1024);
      const uint64_t q_mn = make_smem_desc(smem_u32(sQ), kFbHalf, 1024), do_mn = make_smem_desc(smem_u32(sdO), kFbHalf, 1024);
      // [128 x 128] = A B^T, both K-major in shared memory
      auto product_kk = [&](uint32_t dst, uint64_t a, uint64_t b) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint32_t off = ((k >> 2) * kFbHalf + (k & 3) * 32) >> 4;
          umma_bf16_warp(e, dst, a + off, b + off, idesc_kk, k != 0);
        }
      };
      // [128 x 128] += A B with A in TMEM (16 columns of bf16 pairs in every 32: one group's), B MN-major in shared memory
      auto product_ts = [&](uint32_t dst, uint32_t a, uint64_t b, uint32_t add) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_bf16_ts_warp(e, dst, a + (k >> 1) * 32 + (k & 1) * 8, b + ((k * 2048) >> 4), idesc_km, add | k);
      };
      bool ok = mbar_wait_warp(&sh->kv_full, 0, abort_flag) && mbar_wait_warp(&sh->q_full[0], 0, abort_flag);
      if (ok) {
        tc_fence_after();
        product_kk(tm, k_kk, q_kk);
        umma_commit_warp(e, &sh->s_full);
        ok = mbar_wait_warp(&sh->do_full[0], 0, abort_flag);
      }
      if (ok) {
        tc_fence_after();
        product_kk(tm + 128, v_kk, do_kk);
        umma_commit_warp(e, &sh->dp_full);
      }
      for (int it = 0; ok && it < n_it; ++it) {
        const int s = it & 1, s2 = s ^ 1;
        const uint32_t ph2 = ((it + 1) >> 1) & 1;
        constexpr uint32_t tile = kFbTileBytes >> 4;
        const bool more = it + 1 < n_it;
        // dV += P^T dO, then S of the next step over P^T (the tensor core takes the products of this warp in order)
        if (!mbar_wait_warp(&sh->p_full, it & 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        product_ts(tm + 256, tm, do_mn + s * tile, it != 0);
        umma_commit_warp(e, &sh->do_empty[s]);
        if (more) {
          if (!mbar_wait_warp(&sh->q_full[s2], ph2, abort_flag)) { ok = false; break; }
          tc_fence_after();
          product_kk(tm, k_kk, q_kk + s2 * tile);
          umma_commit_warp(e, &sh->s_full);
        }
        // dK += dS^T Q, then dP of the next step over dS^T
        if (!mbar_wait_warp(&sh->ds_full, it & 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        product_ts(tm + 384, tm + 128, q_mn + s * tile, it != 0);
        umma_commit_warp(e, &sh->q_empty[s]);
        if (more) {
          if (!mbar_wait_warp(&sh->do_full[s2], ph2, abort_flag)) { ok = false; break; }
          tc_fence_after();
          product_kk(tm + 128, v_kk, do_kk + s2 * tile);
          umma_commit_warp(e, &sh->dp_full);
        }
      }
      umma_commit_warp(e, &sh->done);
      if (!ok && e) {
        sh->abort_flag = 1;
        atomicCAS(err, 0, kFbErrMma);
      }
    } else if (warp == 2) {
      // ------------------------------- statistics of the query tiles -------------------------------
      bool ok = true;
      int it = 0;
      for (int g = 0; g < G && ok; ++g) {
        const size_t base = (size_t)(h_first + g) * T;
        for (int i = j; i < i_end; ++i, ++it) {
          const int s = it & 1;
          float l[4], dl[4];
          int st[4];
#pragma unroll
          for (int c = 0; c < 4; ++c) {        // rows past T: their Q and dO are zeros
            const int row = i * kFbTile + c * 32 + lane;
            l[c] = row < T ? fa.lse[base + row] * -1.4426950408889634f : 0.f;
            dl[c] = row < T ? -fa.delta[base + row] * fa.scale : 0.f;
            st[c] = row < T ? fa.row_start[row] : 0x7fffffff;
          }
          if (!mbar_wait_warp(&sh->st_empty[s], ((it >> 1) & 1) ^ 1, abort_flag)) { ok = false; break; }
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            sh->lse2[s][c * 32 + lane] = l[c];
            sh->nds[s][c * 32 + lane] = dl[c];
            sh->start[s][c * 32 + lane] = st[c];
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&sh->st_full[s]);
        }
      }
      if (!ok && lane == 0) {
        sh->abort_flag = 1;
        atomicCAS(err, 0, kFbErrStats);
      }
    }
  } else {
    // ------------------- P / dS / epilogue: thread <-> key -------------------
    setmaxnreg_inc<kFbRegsSoftmax>();
    const int wg = (warp - 4) >> 2;              // queries 32 wg .. of a tile
    const int quad = warp & 3;                   // TMEM lane quadrant this warp may access
    const int r = quad * 32 + lane, key = k0 + r;
    const uint32_t lane_off = (uint32_t)(quad * 32) << 16;
    const uint32_t t_s = tmem_base + lane_off + wg * 32, t_dp = t_s + 128;
    const float scale = fa.scale, scale_log2 = scale * 1.4426950408889634f;
    bool ok = true;
    auto fail = [&]() {
      ok = false;
      sh->abort_flag = 1;
      atomicCAS(err, 0, kFbErrSoftmax);
    };
    int it = 0;
    for (int g = 0; g < G; ++g) {
      // ALiBi: P is recomputed with the forward's bias (slope / scale) * (key - query) of the raw score (a constant of q and k: no
      // gradient)
      const float alibi_s = fa.alibi_slopes != nullptr ? fa.alibi_slopes[h_first + g] / scale : 0.f;
      for (int i = j; i < i_end; ++i, ++it) {
        const int s = it & 1;
        const uint32_t ph = it & 1;
        const int q0 = i * kFbTile;
        if (!mbar_wait(&sh->st_full[s], (it >> 1) & 1, abort_flag)) fail();
        const float* lse2 = sh->lse2[s] + wg * 32;
        const float* nds = sh->nds[s] + wg * 32;
        const int* start = sh->start[s] + wg * 32;
        const bool need_mask = i == j || sh->start[s][min(q0 + kFbTile, T) - 1 - q0] > k0;
        if (!mbar_wait(&sh->s_full, ph, abort_flag)) fail();
        tc_fence_after();
        uint32_t v[32], pk[16];
        tmem_ld_32x32(t_s, v);
        tmem_ld_wait();
        uint32_t seen = 0xffffffffu;
        if (need_mask) {
          // the queries that see the key are those from the key's own row to the end of its document; starts do not decrease
          int n = 0;                           // of 32 queries, those whose document starts at or before the key
#pragma unroll
          for (int b = 16; b > 0; b >>= 1)
            if (start[n + b - 1] <= key) n += b;
          if (n == 31 && start[31] <= key) n = 32;
          seen = fb_bits(key - (q0 + wg * 32), n - 1);
        }
        fb_mask32(v, seen);
        if (fa.alibi_slopes != nullptr) {
          const float d0 = (float)(key - (q0 + wg * 32));
#pragma unroll
          for (int e = 0; e < 32; ++e) v[e] = __float_as_uint(fmaf(alibi_s, d0 - (float)e, __uint_as_float(v[e])));
        }
#pragma unroll
        for (int e = 0; e < 32; e += 4) {
          const float4 off = *reinterpret_cast<const float4*>(lse2 + e);
          const float2 sc = make_float2(scale_log2, scale_log2);
          const float2 a = ffma2(make_float2(__uint_as_float(v[e]), __uint_as_float(v[e + 1])), sc, make_float2(off.x, off.y));
          const float2 b = ffma2(make_float2(__uint_as_float(v[e + 2]), __uint_as_float(v[e + 3])), sc, make_float2(off.z, off.w));
          pk[e / 2] = fb_pack(ex2_approx(a.x), ex2_approx(a.y));
          pk[e / 2 + 1] = fb_pack(ex2_approx(b.x), ex2_approx(b.y));
        }
        tmem_st_32x16(t_s, pk);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh->p_full);
        if (!mbar_wait(&sh->dp_full, ph, abort_flag)) fail();
        tc_fence_after();
        tmem_ld_32x32(t_dp, v);
        tmem_ld_wait();
        fb_ds32(v, pk, scale, [&](int e) { return *reinterpret_cast<const float2*>(nds + 2 * e); }, pk);
        tmem_st_32x16(t_dp, pk);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&sh->ds_full);
          mbar_arrive(&sh->st_empty[s]);
        }
      }
    }
    // ---------------- epilogue: halves of dV (groups 0, 1) and dK (2, 3), through what held Q and dO ----------------
    if (!mbar_wait(&sh->done, 0, abort_flag)) fail();
    tc_fence_after();
    const bool write = __all_sync(0xffffffffu, ok && !*abort_flag);
    const uint32_t t_acc = tmem_base + lane_off + 256 + wg * 64;
    const CUtensorMap* map = wg < 2 ? &tmdV : &tmdK;
    const int col = (wg & 1) * 64;
    uint8_t* stage = sQ + (warp - 4) * 8192;
    if (write && fa.nsplit > 1) {
      // the query-head group is split over CTAs: add to the fp32 sums [2][T, Hk * 128] (dk, dv)
#pragma unroll 1
      for (int c = 0; c < 2; ++c) {
        uint32_t v[32];
        tmem_ld_32x32(t_acc + c * 32, v);
        tmem_ld_wait();
#pragma unroll
        for (int g4 = 0; g4 < 8; ++g4)
          *reinterpret_cast<uint4*>(stage + c * 4096 + lane * 128 + ((g4 ^ (lane & 7)) << 4)) =
              make_uint4(v[g4 * 4], v[g4 * 4 + 1], v[g4 * 4 + 2], v[g4 * 4 + 3]);
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        for (int c = 0; c < 2; ++c) tma_reduce_add_2d(map, stage + c * 4096, kvh * kFbD + col + c * 32, k0 + quad * 32);
        tma_store_commit();
        tma_store_wait_read<0>();
      }
    } else if (write) {
      fb_stage64(t_acc, stage, lane);
      if (lane == 0) {
        tma_store_3d(map, stage, col, kvh, k0 + quad * 32);
        tma_store_commit();
        tma_store_wait_read<0>();
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) {
    // error path: give copies / products still in flight time to land before smem and TMEM go away
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) {
    }
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc<512>(tmem_base);
  }
}

// ------------------------------------------------ queries ------------------------------------------------
struct FbItem {
  int valid, q0, h, kv_lo, n, max_start;       // n key tiles from kv_lo; max_start: document start of the tile's last row
};
struct FbQShared {
  uint64_t q_full, q_empty, do_full, do_empty, k_full[2], k_empty[2], v_full[2], v_empty[2], s_full, s_free, dp_full[2], dq_full;
  // A barrier for even and one for odd steps: dP of a step is there before dS of the step before is waited for, so a warp may be done
  // with a step while another still makes the one before.
  uint64_t ds_full[2];
  uint64_t item_full[2], item_empty[2], claim, claimed;
  alignas(16) uint32_t response[4];
  FbItem item[2];
  uint32_t tmem_base;
  int abort_flag;
};
constexpr int kFbQOps = 6 * kFbTileBytes;       // Q, dO, K x2, V x2
constexpr int kFbQSmem = kFbQOps + 32768 + 1024 + 512;
static_assert(sizeof(FbQShared) <= 512, "");

__global__ void __launch_bounds__(kFbThreads, 1)
flash_bwd_q_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                   const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                   const __grid_constant__ CUtensorMap tmdQ, const __grid_constant__ FbArgs fa) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t *sQ = smem, *sdO = smem + kFbTileBytes, *sK = smem + 2 * kFbTileBytes, *sV = smem + 4 * kFbTileBytes;
  FbQShared* sh = reinterpret_cast<FbQShared*>(smem + kFbQOps + 32768);
  int* const err = fa.err;
  const int T = fa.T;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    mbar_init(&sh->q_full, 1);
    mbar_init(&sh->q_empty, 1);
    mbar_init(&sh->do_full, 1);
    mbar_init(&sh->do_empty, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&sh->k_full[s], 1);
      mbar_init(&sh->k_empty[s], 1);
      mbar_init(&sh->v_full[s], 1);
      mbar_init(&sh->v_empty[s], 1);
      mbar_init(&sh->dp_full[s], 1);
      mbar_init(&sh->ds_full[s], kFbSoftmaxWarps);
      mbar_init(&sh->item_full[s], 1);
      mbar_init(&sh->item_empty[s], 1 + 1 + kFbSoftmaxWarps);   // loader, MMA warp, softmax warps
    }
    mbar_init(&sh->s_full, 1);
    mbar_init(&sh->s_free, kFbSoftmaxWarps);
    mbar_init(&sh->dq_full, 1);
    mbar_init(&sh->claim, 1);
    mbar_init(&sh->claimed, 1);
    sh->abort_flag = *(volatile int*)err;      // an earlier CTA already failed: do not wait on anything
    fence_barrier_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmdO);
  }
  if (warp == 1) tmem_alloc<512>(&sh->tmem_base);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = sh->tmem_base;
  const bool dead_on_arrival = sh->abort_flag != 0;
  volatile int* abort_flag = &sh->abort_flag;

  if (dead_on_arrival) {
    // fall through to the common exit: nothing was issued
  } else if (warp < 4) {
    setmaxnreg_dec<kFbRegsIo>();
    if (warp == 0 && lane == 0) {
      // ------------------------------- TMA loads -------------------------------
      bool ok = true;
      int g = 0;                               // key tiles before the item
      for (int i = 0; ok; ++i) {
        if (!mbar_wait(&sh->item_full[i & 1], (i >> 1) & 1, abort_flag)) { ok = false; break; }
        const FbItem it = sh->item[i & 1];
        mbar_arrive(&sh->item_empty[i & 1]);
        if (!it.valid) break;
        const int x = it.h * kFbD, kx = it.h / (fa.Hq / fa.Hk) * kFbD;
        if (!mbar_wait(&sh->q_empty, (i & 1) ^ 1, abort_flag)) { ok = false; break; }
        mbar_expect_tx(&sh->q_full, kFbTileBytes);
        fb_load_tile(sQ, &tmQ, &sh->q_full, x, it.q0);
        for (int t = 0; t < it.n; ++t) {
          const int s = (g + t) & 1;
          const uint32_t ph = (((g + t) >> 1) & 1) ^ 1;
          if (t == max(it.n - 2, 0)) mbar_arrive(&sh->claim);     // near the end: time to ask for the next item
          if (!mbar_wait(&sh->k_empty[s], ph, abort_flag)) { ok = false; break; }
          mbar_expect_tx(&sh->k_full[s], kFbTileBytes);
          fb_load_tile(sK + s * kFbTileBytes, &tmK, &sh->k_full[s], kx, it.kv_lo + t * kFbTile);
          if (t == 0) {
            if (!mbar_wait(&sh->do_empty, (i & 1) ^ 1, abort_flag)) { ok = false; break; }
            mbar_expect_tx(&sh->do_full, kFbTileBytes);
            fb_load_tile(sdO, &tmdO, &sh->do_full, x, it.q0);
          }
          if (!mbar_wait(&sh->v_empty[s], ph, abort_flag)) { ok = false; break; }
          mbar_expect_tx(&sh->v_full[s], kFbTileBytes);
          fb_load_tile(sV + s * kFbTileBytes, &tmV, &sh->v_full[s], kx, it.kv_lo + t * kFbTile);
        }
        g += it.n;
      }
      if (!ok) {
        sh->abort_flag = 1;
        atomicCAS(err, 0, kFbErrProducer);
      }
    } else if (warp == 1) {
      // ------------------------------- MMA issuer -------------------------------
      constexpr uint32_t idesc_kk = make_idesc_bf16(128, 128, false, false);  // A, B K-major
      constexpr uint32_t idesc_km = make_idesc_bf16(128, 128, false, true);   // A K-major (TMEM), B MN-major
      constexpr uint32_t tile = kFbTileBytes >> 4;
      const uint32_t e = elect_one(), tm = __reduce_or_sync(0xffffffffu, tmem_base);
      const uint64_t q_kk = make_smem_desc(smem_u32(sQ), 16, 1024), do_kk = make_smem_desc(smem_u32(sdO), 16, 1024);
      const uint64_t k_kk = make_smem_desc(smem_u32(sK), 16, 1024), v_kk = make_smem_desc(smem_u32(sV), 16, 1024);
      const uint64_t k_mn = make_smem_desc(smem_u32(sK), kFbHalf, 1024);
      bool ok = true;
      int g = 0;                               // steps so far
      // S and dP of step g: S once the scores of the step before have been read, dP over the dS of two steps before
      auto scores = [&](int item, bool first, bool last) -> bool {
        const int s = g & 1;
        const uint32_t ph = (g >> 1) & 1;
        if (first && !mbar_wait_warp(&sh->q_full, item & 1, abort_flag)) return false;
        if (!mbar_wait_warp(&sh->k_full[s], ph, abort_flag)) return false;
        if (g > 0 && !mbar_wait_warp(&sh->s_free, (g - 1) & 1, abort_flag)) return false;
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint32_t off = ((k >> 2) * kFbHalf + (k & 3) * 32) >> 4;
          umma_bf16_warp(e, tm, q_kk + off, k_kk + s * tile + off, idesc_kk, k != 0);
        }
        umma_commit_warp(e, &sh->s_full);
        if (last) umma_commit_warp(e, &sh->q_empty);
        if (first && !mbar_wait_warp(&sh->do_full, item & 1, abort_flag)) return false;
        if (!mbar_wait_warp(&sh->v_full[s], ph, abort_flag)) return false;
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint32_t off = ((k >> 2) * kFbHalf + (k & 3) * 32) >> 4;
          umma_bf16_warp(e, tm + 128 + s * 128, do_kk + off, v_kk + s * tile + off, idesc_kk, k != 0);
        }
        umma_commit_warp(e, &sh->dp_full[s]);
        umma_commit_warp(e, &sh->v_empty[s]);
        if (last) umma_commit_warp(e, &sh->do_empty);
        return true;
      };
      for (int i = 0; ok; ++i) {
        ok = mbar_wait_warp(&sh->item_full[i & 1], (i >> 1) & 1, abort_flag);
        if (!ok) break;
        const bool valid = warp_uniform(sh->item[i & 1].valid != 0);
        const int n = sh->item[i & 1].n;
        __syncwarp();
        if (e) mbar_arrive(&sh->item_empty[i & 1]);
        if (!valid) break;
        ok = scores(i, true, warp_uniform(n == 1));
        for (int t = 0; warp_uniform(t < n) && ok; ++t) {
          const int s = g & 1;
          const uint32_t ph = (g >> 1) & 1;
          const bool more = warp_uniform(t + 1 < n);
          ++g;
          if (more) ok = scores(i, false, warp_uniform(t + 2 == n));
          // dQ += dS K
          ok = ok && mbar_wait_warp(&sh->ds_full[s], ph, abort_flag);
          if (!ok) break;
          tc_fence_after();
          const uint64_t b = k_mn + s * tile;
          const uint32_t add = t != 0;
#pragma unroll
          for (int k = 0; k < 8; ++k)
            umma_bf16_ts_warp(e, tm + 384, tm + 128 + s * 128 + (k >> 1) * 32 + (k & 1) * 8, b + ((k * 2048) >> 4), idesc_km, add | k);
          umma_commit_warp(e, &sh->k_empty[s]);
          if (!more) umma_commit_warp(e, &sh->dq_full);
        }
      }
      if (!ok && e) {
        sh->abort_flag = 1;
        atomicCAS(err, 0, kFbErrMma);
      }
    } else if (warp == 2 && lane == 0) {
      // ------------------------------- work items: the CTA's own index, then those of CTAs that have not started ------------
      const int n_qt = (T + kFbTile - 1) / kFbTile;
      bool ok = true;
      int index = blockIdx.x;
      for (int i = 0; ok; ++i) {
        FbItem it{};
        if (i > 0) {
          if (!mbar_wait(&sh->claim, (i - 1) & 1, abort_flag)) { ok = false; break; }
          mbar_expect_tx(&sh->claimed, 16);
          clc_try_cancel(sh->response, &sh->claimed);
          if (!mbar_wait(&sh->claimed, (i - 1) & 1, abort_flag)) { ok = false; break; }
          index = clc_first_cta(sh->response);
          fence_proxy_async_smem();
        }
        it.valid = index >= 0;
        if (it.valid) {                        // the longest walks of all heads first
          it.q0 = (n_qt - 1 - index / fa.Hq) * kFbTile;
          it.h = index % fa.Hq;
          const int last = min(it.q0 + kFbTile, T) - 1;
          it.kv_lo = fa.row_start[it.q0];
          it.max_start = fa.row_start[last];
          it.n = (last - it.kv_lo) / kFbTile + 1;
        }
        if (!mbar_wait(&sh->item_empty[i & 1], ((i >> 1) & 1) ^ 1, abort_flag)) { ok = false; break; }
        sh->item[i & 1] = it;
        mbar_arrive(&sh->item_full[i & 1]);
        if (!it.valid) break;
      }
      if (!ok) {
        sh->abort_flag = 1;
        atomicCAS(err, 0, kFbErrStats);
      }
    }
  } else {
    // ------------------- P / dS / epilogue: thread <-> query -------------------
    setmaxnreg_inc<kFbRegsSoftmax>();
    const int wg = (warp - 4) >> 2;              // keys 32 wg .. of a tile
    const int quad = warp & 3;
    const int r = quad * 32 + lane;
    const uint32_t lane_off = (uint32_t)(quad * 32) << 16;
    const uint32_t t_s = tmem_base + lane_off + wg * 32;
    const float scale = fa.scale, scale_log2 = scale * 1.4426950408889634f;
    uint8_t* stage = smem + kFbQOps + ((warp - 4) & 7) * 4096;
    bool ok = true;
    auto fail = [&]() {
      ok = false;
      sh->abort_flag = 1;
      atomicCAS(err, 0, kFbErrSoftmax);
    };
    int g = 0;                                   // steps so far
    for (int i = 0;; ++i) {
      if (!mbar_wait(&sh->item_full[i & 1], (i >> 1) & 1, abort_flag)) fail();
      if (__any_sync(0xffffffffu, !ok)) break;
      const FbItem it = sh->item[i & 1];
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh->item_empty[i & 1]);
      if (!it.valid) break;
      const int row = it.q0 + r;
      const bool row_valid = row < T;
      const int my_start = row_valid ? fa.row_start[row] : 0x7fffffff;
      const float nl = row_valid ? fa.lse[(size_t)it.h * T + row] * -1.4426950408889634f : 0.f;
      const float nd = row_valid ? -fa.delta[(size_t)it.h * T + row] * scale : 0.f;
      const float alibi_s = fa.alibi_slopes != nullptr ? fa.alibi_slopes[it.h] / scale : 0.f;
      for (int t = 0; t < it.n; ++t, ++g) {
        const int k0 = it.kv_lo + t * kFbTile, kc = k0 + wg * 32;
        const uint32_t t_dp = t_s + 128 + (g & 1) * 128;
        const bool need_mask = k0 + kFbTile - 1 > it.q0 || it.max_start > k0;
        if (!mbar_wait(&sh->s_full, g & 1, abort_flag)) fail();
        tc_fence_after();
        uint32_t v[32], pk[16];
        tmem_ld_32x32(t_s, v);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh->s_free);
        fb_mask32(v, need_mask ? fb_bits(my_start - kc, row - kc) : 0xffffffffu);
        if (fa.alibi_slopes != nullptr) {
          const float d0 = (float)(kc - row);
#pragma unroll
          for (int e = 0; e < 32; ++e) v[e] = __float_as_uint(fmaf(alibi_s, d0 + (float)e, __uint_as_float(v[e])));
        }
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          const float2 x = ffma2(make_float2(__uint_as_float(v[e]), __uint_as_float(v[e + 1])), make_float2(scale_log2, scale_log2),
                                 make_float2(nl, nl));
          pk[e / 2] = fb_pack(ex2_approx(x.x), ex2_approx(x.y));
        }
        if (!mbar_wait(&sh->dp_full[g & 1], (g >> 1) & 1, abort_flag)) fail();
        tc_fence_after();
        tmem_ld_32x32(t_dp, v);
        tmem_ld_wait();
        fb_ds32(v, pk, scale, [&](int) { return make_float2(nd, nd); }, pk);
        tmem_st_32x16(t_dp, pk);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh->ds_full[g & 1]);
      }
      // ---------------- epilogue: 32 rows x 64 columns a warp, from groups 0 and 1 (the others go on) ----------------
      if (wg < 2) {
        if (!mbar_wait(&sh->dq_full, i & 1, abort_flag)) fail();
        tc_fence_after();
        const bool write = __all_sync(0xffffffffu, ok && !*abort_flag);
        if (lane == 0) tma_store_wait_read<0>();   // of the item before
        __syncwarp();
        fb_stage64(tmem_base + lane_off + 384 + wg * 64, stage, lane);
        tc_fence_before();
        if (lane == 0 && write) {
          tma_store_3d(&tmdQ, stage, wg * 64, it.h, it.q0 + quad * 32);
          tma_store_commit();
        }
      }
    }
    if (lane == 0) tma_store_wait_read<0>();
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) {
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) {
    }
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc<512>(tmem_base);
  }
}

// delta[h, t] = sum_d dO[t, h, d] * O[t, h, d]; 16 lanes a row, four rows one after the other: eight 16-byte loads in flight a lane.
__global__ void flash_bwd_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ dout,
                                       float* __restrict__ delta, int T, int Hq) {
  const long long first = ((long long)blockIdx.x * 256 + threadIdx.x) / 16 * 4, n = (long long)T * Hq;
  const int lane = threadIdx.x & 15;
  bf16x8 a[4], b[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const long long w = min(first + i, n - 1);
    a[i] = reinterpret_cast<const bf16x8*>(o + w * kFbD)[lane];
    b[i] = reinterpret_cast<const bf16x8*>(dout + w * kFbD)[lane];
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float x[8], y[8], s = 0.f;
    unpack8(a[i], x);
    unpack8(b[i], y);
#pragma unroll
    for (int c = 0; c < 8; ++c) s = fmaf(x[c], y[c], s);
#pragma unroll
    for (int c = 8; c > 0; c >>= 1) s += __shfl_xor_sync(0xffffffffu, s, c);
    const long long w = first + i;
    if (lane == 0 && w < n) delta[(size_t)(w % Hq) * T + w / Hq] = s;
  }
}

// dk, dv (bf16, rows of `stride` elements) = acc (fp32 [2, T, W]); 8 elements per thread.
__global__ void flash_bwd_convert_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ dk, __nv_bfloat16* __restrict__ dv,
                                         int T, int W, int stride) {
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int vec_per_row = W / 8;
  if (idx >= (size_t)T * vec_per_row) return;
  const int t = idx / vec_per_row, c = idx % vec_per_row;
  const float4* src = reinterpret_cast<const float4*>(acc + ((size_t)blockIdx.y * T + t) * W);
  const float4 x = src[2 * c], y = src[2 * c + 1];
  const float f[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
  reinterpret_cast<bf16x8*>((blockIdx.y == 0 ? dk : dv) + (size_t)t * stride)[c] = pack8(f);
}

int make_tmap_bf16_2d(CUtensorMap* map, const void* ptr, uint64_t inner, uint64_t outer, uint64_t row_stride_bytes,
                      uint32_t box_inner, uint32_t box_outer);
int make_tmap_f32_2d(CUtensorMap* map, const void* ptr, uint64_t inner, uint64_t outer, uint64_t row_stride_bytes,
                     uint32_t box_inner, uint32_t box_outer);
int make_tmap_bf16_heads(CUtensorMap* map, const void* ptr, uint64_t dim, uint64_t heads, uint64_t rows,
                         uint64_t row_stride_bytes, uint32_t box_dim, uint32_t box_rows, uint64_t head_stride_bytes = 0);

}  // namespace ell

using namespace ell;

// q [T, Hq, 128], k / v [T, Hk, 128] (row strides q_stride / kv_stride elements, views into a packed QKV
// buffer are fine); out, dout [T, Hq, 128] contiguous, on 16-byte places; lse [Hq, T] from the forward.
// Outputs: dq [T, Hq, 128] (row stride dq_stride), dk / dv [T, Hk, 128] (row stride dkv_stride) - views into
// one packed dQKV buffer are fine.  Scratch: delta fp32 [Hq, T],
// dkv_acc fp32 [2, T, Hk*128] (GQA only, may be null: used when the head group is split over CTAs).
ELL_API int ell_flash_attn_bwd(const void* q, const void* k, const void* v, const void* out, const void* dout,
                               const float* lse, const int* row_start, void* dq, void* dk, void* dv,
                               float* delta, float* dkv_acc, int T, int Hq, int Hk, int q_stride, int kv_stride, int dq_stride,
                               int dkv_stride, float scale, const float* alibi_slopes, int* err, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (Hq % Hk) return -2;
  if ((dq_stride % 8) || (dkv_stride % 8) || ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(dout)) & 15)) return -3;
  const int n_kt = (T + kFbTile - 1) / kFbTile;
  // few kv heads and a short sequence leave SMs idle: split each query-head group over CTAs
  const int nsplit = (Hq > Hk && dkv_acc != nullptr && Hk * n_kt < 2 * kNumSMs) ? Hq / Hk : 1;
  const int Wk = Hk * kFbD;
  CUtensorMap tq, tk, tv, tdo, tdq, tdk, tdv;
  int rc = make_tmap_bf16_2d(&tq, q, (uint64_t)Hq * kFbD, (uint64_t)T, (uint64_t)q_stride * 2, 64, 128);
  if (!rc) rc = make_tmap_bf16_2d(&tk, k, (uint64_t)Wk, (uint64_t)T, (uint64_t)kv_stride * 2, 64, 128);
  if (!rc) rc = make_tmap_bf16_2d(&tv, v, (uint64_t)Wk, (uint64_t)T, (uint64_t)kv_stride * 2, 64, 128);
  if (!rc) rc = make_tmap_bf16_2d(&tdo, dout, (uint64_t)Hq * kFbD, (uint64_t)T, (uint64_t)Hq * kFbD * 2, 64, 128);
  if (!rc) rc = make_tmap_bf16_heads(&tdq, dq, kFbD, Hq, T, (uint64_t)dq_stride * 2, 64, 32);
  if (nsplit > 1) {
    if (!rc) rc = make_tmap_f32_2d(&tdk, dkv_acc, (uint64_t)Wk, (uint64_t)T, (uint64_t)Wk * 4, 32, 32);
    if (!rc) rc = make_tmap_f32_2d(&tdv, dkv_acc + (size_t)T * Wk, (uint64_t)Wk, (uint64_t)T, (uint64_t)Wk * 4, 32, 32);
  } else {
    if (!rc) rc = make_tmap_bf16_heads(&tdk, dk, kFbD, Hk, T, (uint64_t)dkv_stride * 2, 64, 32);
    if (!rc) rc = make_tmap_bf16_heads(&tdv, dv, kFbD, Hk, T, (uint64_t)dkv_stride * 2, 64, 32);
  }
  if (rc) return rc;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(flash_bwd_kv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFbKvSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(flash_bwd_q_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFbQSmem);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  if (nsplit > 1) {
    cudaError_t e = cudaMemsetAsync(dkv_acc, 0, (size_t)2 * T * Wk * sizeof(float), stream);
    if (e != cudaSuccess) return (int)e;
  }
  const long long rows = (long long)T * Hq, grid_q = (long long)n_kt * Hq;
  if (grid_q > 0x7fffffff) return -2;
  flash_bwd_delta_kernel<<<(unsigned)((rows + 63) / 64), 256, 0, stream>>>((const __nv_bfloat16*)out, (const __nv_bfloat16*)dout, delta,
                                                                           T, Hq);
  const FbArgs fa{lse, delta, row_start, T, Hq, Hk, nsplit, scale, alibi_slopes, err};
  flash_bwd_kv_kernel<<<dim3(Hk * nsplit, n_kt), kFbThreads, kFbKvSmem, stream>>>(tq, tk, tv, tdo, tdk, tdv, fa);
  if (nsplit > 1) {
    const size_t n = (size_t)T * (Wk / 8);
    flash_bwd_convert_kernel<<<dim3((unsigned)((n + 255) / 256), 2), 256, 0, stream>>>(dkv_acc, (__nv_bfloat16*)dk, (__nv_bfloat16*)dv, T,
                                                                                      Wk, dkv_stride);
  }
  flash_bwd_q_kernel<<<(unsigned)grid_q, kFbThreads, kFbQSmem, stream>>>(tq, tk, tv, tdo, tdq, fa);
  return launch_status();
}
