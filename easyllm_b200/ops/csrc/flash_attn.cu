// Causal flash attention forward on tcgen05 / TMEM for sm_100a: packed variable-length
// documents, MHA and GQA, key and value heads of up to 128 (multiples of 8, sizes of their own), bf16 in/out, fp32
// softmax with an optional learned sink per head in the denominator.
//
// A work item is a pair of adjacent 128-query tiles of one query head.  A CTA takes the item of its own index and then, one at a time
// and near the end of the one before, items of CTAs that have not started (cluster launch control); 384 threads:
//   warp 0     TMA: the Q tiles of an item, K tiles (128 keys) and V tiles through rings of two stages
//   warps 1, 3 one per query tile t: for every key tile j that t sees, S_t = Q_t·K_jᵀ (128x128x128) and O_t += P_t·V_j (P from TMEM, V
//              read in place as an MN-major operand).  The whole warp walks the loop, see sm100.cuh.
//              TMEM columns: S_0 | P_0 0-127, S_1 | P_1 128-255, O_0 256-383, O_1 384-511.
//   warp 2     work items: which one, the key tiles that each of its query tiles sees
//   warps 4-7 / 8-11  one softmax group per query tile: thread r owns query row r (its TMEM lane), so row
//              max / row sum need no shuffles.  The whole S row is pulled into registers at once, exp2 with the scale folded into one
//              FMA, P written as bf16 pairs over the first half of the scores' columns (the product with V starts on the first half of
//              P); the O accumulator is rescaled only when a row maximum grew by more than 2^8 (stale-max trick: the final
//              1/l normalisation makes it exact).  Rows leave through shared memory and TMA stores.
// The two tiles run on their own and so fall into alternation: one's softmax (2300 cycles a step, 1024 of them the special-function
// unit's) beside the other's products (2 x 512).  What this replaced kept P in shared memory, whose bandwidth the two operands and P
// filled, issued from one lane's branch (90 to 210 cycles a product that takes 65, see sm100.cuh), and left the SM empty between
// items: start, masked diagonal, 4000 cycles of row-wise stores.  us, one B200, inputs not in L2, before -> now: 4096 tokens, 32 heads
// 196 -> 153 (0.90 PFLOP/s); 8 documents of 512, 32 heads on 8 92 -> 40; 3001 tokens in 7 documents, 16 on 4 54 -> 32; 77 tokens 15.3 -> 11.3
// (launch included); latent keys of 128 + 64, 4096 tokens, 32 heads, a window of 1024 181 -> 118.
// A single warp that took whichever tile could go cost 500 cycles a turn of its loop in looking around (4096 tokens 165 us).
// Documents: row_start[t] is the first token of the document that token t belongs to; key j is
// visible to query i iff row_start[i] <= j <= i, so tiles may straddle document boundaries.
// ALiBi: with per-head slopes the score of (query i, key j) gets the bias slope_h * (j - i) before the softmax
// (llm/models/hf_models/baichuan2/model_13b/modeling_baichuan.py:63-73 builds the same bias as a mask tensor).
//
// Head sizes below 128: the tensor maps are [dim, heads, rows], so a 64-column box that reaches past a head's end is
// zero-filled by the TMA unit; the score product runs ceil(dim / 16) k-steps and P·V is ceil(vdim / 16) * 16 wide.
//
// Keys in two parts (latent attention): a head's key is a part of its own followed by a part shared by all heads, read
// from its own rows; the query row holds both.  Each part fills 64-column chunks of the tiles, so nothing is assembled in
// memory.  Keys of more than two chunks (e.g. 128 + 64) use key tiles of 64 instead of 128 rows to fit shared memory.
// A window limits row i to the keys i - window + 1 .. i; a gate multiplies head h's output of row i by sigmoid(gate[i][h]).
//
// Replaces flash_attn_varlen_{qkv,kv}packed_func of the reference
// (llm/models/mg_models/llama/transformer.py:65-143).
#include "common.cuh"
#include "sm100.cuh"

namespace ell {
using namespace sm100;

constexpr int kFaThreads = 384;
constexpr int kFaM = 128, kFaN = 128, kFaD = 128;
// Registers a thread after the split of the launch's 168 x 384: a softmax thread holds a whole row of scores.
constexpr int kFaRegsIo = 104, kFaRegsSoftmax = 200;
// Shared memory of a configuration: KN keys a tile, NC 64-column chunks a query / key row.
template <int KN, int NC>
struct FaCfg {
  static constexpr int kQChunk = kFaM * 128;           // [128 rows x 64 columns] bf16, 128-byte swizzle rows
  static constexpr int kKChunk = KN * 128;
  static constexpr int kQBytes = NC * kQChunk, kKBytes = NC * kKChunk;
  static constexpr int kVBytes = 2 * kKChunk;          // value heads of up to 128
  static constexpr int kOps = 2 * kQBytes + 2 * kKBytes + 2 * kVBytes;   // Q x2, K x2, V x2
  static constexpr int kBars = kOps + 32768;           // between them the output rows on their way out
  static constexpr int kSmemBytes = kBars + 1024 + 640;
  static_assert(kSmemBytes <= 232448, "");
  static constexpr int kFirst = KN > 64 ? 64 : 32;     // keys of the first part of P
};
constexpr float kFaRescaleThreshold = 8.0f;   // log2 units

// One work item: a pair of query tiles of one head.  jlo / n: the key tiles [jlo, n) that query tile t walks.
struct FaItem {
  int valid, q0, h, kv_lo, jlo[2], n[2], max_start[2];
};

struct FaShared {
  uint64_t q_full[2], q_empty[2], k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[2], p_first[2], p_full[2], o_full[2];
  uint64_t item_full[2], item_empty[2], claim, claimed;
  alignas(16) uint32_t response[4];
  FaItem item[2];
  uint32_t tmem_base;
  int abort_flag;
};

enum FaErr { kFaErrProducer = 11, kFaErrMma = 12, kFaErrSoftmax = 13, kFaErrItems = 17 };

// Tile plan of the forward kernel, __host__ __device__ so that ell_flash_fwd_plan can run the same arithmetic on the
// host for a CPU test.  A query tile starting at row `first` walks key tiles of kFaN keys from kv_lo (the document
// start of the first row of the CTA's tile pair) up to the tile's last row.
__host__ __device__ __forceinline__ int fa_num_kv_tiles(int first, int T, int kv_lo, int kn = kFaN) {
  const int last = (first + kFaM < T ? first + kFaM : T) - 1;
  return first < T ? (last + 1 - kv_lo + kn - 1) / kn : 0;
}

// First key row `row` sees: the start of its document, or of its window.
__host__ __device__ __forceinline__ int fa_first_key(int row, int doc_start, int window) {
  const int w = row - window + 1;
  return w > doc_start ? w : doc_start;
}

// First key tile, counted from kv_lo, with a key that a row whose first key is `first_key` sees (n: none).
__host__ __device__ __forceinline__ int fa_first_kv_tile(int first_key, int kv_lo, int n, int kn = kFaN) {
  const int j = (first_key - kv_lo) / kn;
  return j < n ? j : n;
}

// A key tile starting at k0 needs no per-element mask when every key in it precedes (or is) the tile's first query
// row and no row of the query tile starts its document (or window) after k0.
__host__ __device__ __forceinline__ bool fa_tile_needs_mask(int k0, int tile_first, int max_row_start, int kn = kFaN) {
  return (k0 + kn - 1 > tile_first) || (k0 < max_row_start);
}

struct FaArgs {
  __nv_bfloat16* out;
  float* lse;
  const int* row_start;
  int T, Hq, Hk, d, d2, dv;             // d2: size of the shared key part (0: none)
  int window;                           // keys a row sees at most (INT_MAX: all)
  float scale_log2;
  const float *alibi_slopes, *sink;
  const __nv_bfloat16* gate;            // [T, ldg] or null
  int ldg;
  int* err;
  int head_group;                       // heads whose CTAs are walked together (set at launch)
};

// Query heads whose CTAs come together, in the order of their work.  Head by head, the last head's long walks started last and left
// SMs idle: 30 % of them for 32 heads over 4096 tokens, 233 us where this order took 198.  As many heads as have their keys and values
// in kFaGroupBytes, so that the walks of a group still meet them in L2.
constexpr long long kFaGroupBytes = 64ll << 20;
static int fa_head_group(int T, int Hq, int Hk, int d, int dv) {
  const long long n = kFaGroupBytes * (Hq / Hk) / ((long long)T * (d + dv) * 2);
  return n < 1 ? 1 : (n < Hq ? (int)n : Hq);
}

static_assert(sizeof(FaShared) <= 640, "");

template <int KN, int NC>
__global__ void __launch_bounds__(kFaThreads, 1)
flash_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmQ2,
                 const __grid_constant__ CUtensorMap tmK2, const __grid_constant__ CUtensorMap tmO,
                 const __grid_constant__ FaArgs fa) {
  using Cfg = FaCfg<KN, NC>;
  int* const err = fa.err;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sQ = smem;                          // 2 query tiles
  uint8_t* sK = sQ + 2 * Cfg::kQBytes;         // 2 stages
  uint8_t* sV = sK + 2 * Cfg::kKBytes;         // 2 stages
  FaShared* sh = reinterpret_cast<FaShared*>(smem + Cfg::kBars);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int d = fa.d, dv = fa.dv;
  // chunks of the head's own key part, of both parts, of a value
  const int n1 = (d + 63) / 64, n_chunks = n1 + (fa.d2 + 63) / 64;
  const bool wide_v = dv > 64;

  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&sh->q_full[s], 1);
      mbar_init(&sh->q_empty[s], 1);
      mbar_init(&sh->k_full[s], 1);
      mbar_init(&sh->k_empty[s], 2);           // one from each tile's MMA warp
      mbar_init(&sh->v_full[s], 1);
      mbar_init(&sh->v_empty[s], 2);
      mbar_init(&sh->s_full[s], 1);
      mbar_init(&sh->p_first[s], 4);
      mbar_init(&sh->p_full[s], 4);
      mbar_init(&sh->o_full[s], 1);
      mbar_init(&sh->item_full[s], 1);
      mbar_init(&sh->item_empty[s], 1 + 2 + 8);   // loader, MMA warps, softmax warps
    }
    mbar_init(&sh->claim, 1);
    mbar_init(&sh->claimed, 1);
    sh->abort_flag = *(volatile int*)err;      // an earlier CTA already failed: do not wait on anything
    fence_barrier_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
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
    setmaxnreg_dec<kFaRegsIo>();
    if (warp == 0 && lane == 0) {
      // ------------------------------- TMA loads -------------------------------
      bool ok = true;
      int nq[2] = {0, 0}, g = 0;               // query tiles loaded per slot, key tiles loaded
      for (int i = 0; ok; ++i) {
        if (!mbar_wait(&sh->item_full[i & 1], (i >> 1) & 1, abort_flag)) { ok = false; break; }
        const FaItem it = sh->item[i & 1];
        mbar_arrive(&sh->item_empty[i & 1]);
        if (!it.valid) break;
        const int kvh = it.h / (fa.Hq / fa.Hk), n = max(it.n[0], it.n[1]);
        auto load_q = [&](int t) -> bool {     // rows past T are zero-filled by the TMA unit
          if (it.n[t] <= it.jlo[t]) return true;
          if (!mbar_wait(&sh->q_empty[t], (nq[t] & 1) ^ 1, abort_flag)) return false;
          ++nq[t];
          mbar_expect_tx(&sh->q_full[t], n_chunks * Cfg::kQChunk);
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            if (c >= n_chunks) break;
            tma_load_3d(sQ + t * Cfg::kQBytes + c * Cfg::kQChunk, c < n1 ? &tmQ : &tmQ2, &sh->q_full[t],
                        (c < n1 ? c : c - n1) * 64, it.h, it.q0 + t * kFaM);
          }
          return true;
        };
        auto load_k = [&](int j) -> bool {
          const int s = (g + j) & 1;
          if (!mbar_wait(&sh->k_empty[s], (((g + j) >> 1) & 1) ^ 1, abort_flag)) return false;
          mbar_expect_tx(&sh->k_full[s], n_chunks * Cfg::kKChunk);
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            if (c >= n_chunks) break;
            tma_load_3d(sK + s * Cfg::kKBytes + c * Cfg::kKChunk, c < n1 ? &tmK : &tmK2, &sh->k_full[s],
                        (c < n1 ? c : c - n1) * 64, c < n1 ? kvh : 0, it.kv_lo + j * KN);
          }
          return true;
        };
        ok = load_q(0) && load_k(0) && load_q(1);
        for (int j = 0; j < n && ok; ++j) {
          if (j == max(n - 2, 0)) mbar_arrive(&sh->claim);    // near the end: time to ask for the next item
          if (j + 1 < n && !load_k(j + 1)) { ok = false; break; }
          const int s = (g + j) & 1;
          if (!mbar_wait(&sh->v_empty[s], (((g + j) >> 1) & 1) ^ 1, abort_flag)) { ok = false; break; }
          mbar_expect_tx(&sh->v_full[s], wide_v ? Cfg::kVBytes : Cfg::kKChunk);
          const int k0 = it.kv_lo + j * KN;
          tma_load_3d(sV + s * Cfg::kVBytes, &tmV, &sh->v_full[s], 0, kvh, k0);
          if (wide_v) tma_load_3d(sV + s * Cfg::kVBytes + Cfg::kKChunk, &tmV, &sh->v_full[s], 64, kvh, k0);
        }
        g += n;
      }
      if (!ok) {
        sh->abort_flag = 1;
        atomicCAS(err, 0, kFaErrProducer);
      }
    } else if (warp != 2 && warp != 0) {
      // ------------------------------- MMA issuers: one warp per query tile (one lane's instructions) -----------------------
      // A warp for each tile, so that a tile that ends its item, masks its diagonal or writes its rows does not hold up the other
      // one; the rings of two stages let one be a step ahead.
      constexpr uint32_t idesc_s = make_idesc_bf16(128, KN, false, false);
      const uint32_t idesc_o = make_idesc_bf16(128, (dv + 15) / 16 * 16, false, true);
      const int t = warp >> 1;
      const uint32_t e = elect_one(), tm_s = __reduce_or_sync(0xffffffffu, tmem_base) + t * 128, tm_o = tm_s + 256;
      const uint64_t q_desc = make_smem_desc(smem_u32(sQ), 16, 1024) + t * (Cfg::kQBytes >> 4);
      const uint64_t k_desc = make_smem_desc(smem_u32(sK), 16, 1024), v_desc = make_smem_desc(smem_u32(sV), Cfg::kKChunk, 1024);
      const bool all_steps = n_chunks == NC && d % 64 == 0 && fa.d2 % 64 == 0;
      bool ok = true;
      uint32_t nq = 0, np = 0;                 // query tiles / score tiles so far
      int gk = 0;                              // key tiles before the item
      // S = Q K_j^T goes into the columns of P of the step before: that product was issued earlier by this warp (the tensor core takes
      // them in order), and its P came from the threads that had read the scores before
      auto scores = [&](int g, bool first, bool last) -> bool {
        const int s = g & 1;
        if (first && !mbar_wait_warp(&sh->q_full[t], nq++ & 1, abort_flag)) return false;
        if (!mbar_wait_warp(&sh->k_full[s], (g >> 1) & 1, abort_flag)) return false;
        tc_fence_after();
        const uint64_t kd = k_desc + s * (Cfg::kKBytes >> 4);
        if (all_steps) {
#pragma unroll
          for (int k = 0; k < 4 * NC; ++k)
            umma_bf16_warp(e, tm_s, q_desc + (((k >> 2) * Cfg::kQChunk + (k & 3) * 32) >> 4),
                           kd + (((k >> 2) * Cfg::kKChunk + (k & 3) * 32) >> 4), idesc_s, k != 0);
        } else {
#pragma unroll 1
          for (int c = 0; c < n_chunks; ++c) {
            const int steps = ((c < n1 ? d - c * 64 : fa.d2 - (c - n1) * 64) + 15) / 16;   // past the part: zeros
#pragma unroll 1
            for (int k = 0; k < min(steps, 4); ++k)
              umma_bf16_warp(e, tm_s, q_desc + ((c * Cfg::kQChunk + k * 32) >> 4), kd + ((c * Cfg::kKChunk + k * 32) >> 4), idesc_s,
                             (c | k) != 0);
          }
        }
        umma_commit_warp(e, &sh->s_full[t]);
        umma_commit_warp(e, &sh->k_empty[s]);
        if (last) umma_commit_warp(e, &sh->q_empty[t]);
        return true;
      };
      for (int i = 0; ok; ++i) {
        ok = mbar_wait_warp(&sh->item_full[i & 1], (i >> 1) & 1, abort_flag);
        if (!ok) break;
        const FaItem* it = &sh->item[i & 1];
        const bool valid = warp_uniform(it->valid != 0);
        const int lo = it->jlo[t], hi = it->n[t], n = max(it->n[0], it->n[1]);
        __syncwarp();
        if (e) mbar_arrive(&sh->item_empty[i & 1]);
        if (!valid) break;
        for (int j = 0; warp_uniform(j < n) && ok; ++j) {
          const int s = (gk + j) & 1;
          if (warp_uniform(j < lo || j >= hi)) {           // a key tile that only the other query tile walks
            ok = mbar_wait_warp(&sh->k_full[s], ((gk + j) >> 1) & 1, abort_flag) &&
                 mbar_wait_warp(&sh->v_full[s], ((gk + j) >> 1) & 1, abort_flag);
            if (ok && e) {
              mbar_arrive(&sh->k_empty[s]);
              mbar_arrive(&sh->v_empty[s]);
            }
            __syncwarp();
            continue;
          }
          const bool first = warp_uniform(j == lo), last = warp_uniform(j == hi - 1);
          if (first) ok = scores(gk + j, true, last);
          if (ok) ok = mbar_wait_warp(&sh->v_full[s], ((gk + j) >> 1) & 1, abort_flag) &&
                       mbar_wait_warp(&sh->p_first[t], np & 1, abort_flag);
          if (!ok) break;
          tc_fence_after();
          const uint64_t vd = v_desc + s * (Cfg::kVBytes >> 4);
          const uint32_t add = first ? 0 : 1;
#pragma unroll
          for (int k = 0; k < Cfg::kFirst / 16; ++k)
            umma_bf16_ts_warp(e, tm_o, tm_s + k * 8, vd + ((k * 2048) >> 4), idesc_o, add | k);
          ok = mbar_wait_warp(&sh->p_full[t], np++ & 1, abort_flag);
          if (!ok) break;
          tc_fence_after();
#pragma unroll
          for (int k = Cfg::kFirst / 16; k < KN / 16; ++k)
            umma_bf16_ts_warp(e, tm_o, tm_s + k * 8, vd + ((k * 2048) >> 4), idesc_o, 1);
          umma_commit_warp(e, &sh->v_empty[s]);
          if (last) umma_commit_warp(e, &sh->o_full[t]);
          else ok = scores(gk + j + 1, false, warp_uniform(j + 1 == hi - 1));
        }
        gk += n;
      }
      if (!ok && e) {
        sh->abort_flag = 1;
        atomicCAS(err, 0, kFaErrMma);
      }
    } else if (warp == 2 && lane == 0) {
      // ------------------------------- work items -------------------------------
      // The CTA's own index first, then those of CTAs that have not started: one at a time, when the loads of the item before
      // near their end, so that the last items go to whoever is free.
      const int n_pairs = (fa.T + 2 * kFaM - 1) / (2 * kFaM);
      bool ok = true;
      int index = blockIdx.x;
      for (int i = 0; ok; ++i) {
        FaItem it{};
        if (i > 0) {
          if (!mbar_wait(&sh->claim, (i - 1) & 1, abort_flag)) { ok = false; break; }
          mbar_expect_tx(&sh->claimed, 16);
          clc_try_cancel(sh->response, &sh->claimed);
          if (!mbar_wait(&sh->claimed, (i - 1) & 1, abort_flag)) { ok = false; break; }
          index = clc_first_cta(sh->response);
          fence_proxy_async_smem();
        }
        it.valid = index >= 0;
        if (it.valid) {
          // the heaviest (latest) pairs of a group of heads first
          const int group = index / (fa.head_group * n_pairs), in_group = index - group * fa.head_group * n_pairs;
          const int heads = min(fa.head_group, fa.Hq - group * fa.head_group);
          it.q0 = (n_pairs - 1 - in_group / heads) * 2 * kFaM;
          it.h = group * fa.head_group + in_group % heads;
          int first[2], last[2];
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            first[t] = min(it.q0 + t * kFaM, fa.T - 1);
            last[t] = min(it.q0 + (t + 1) * kFaM, fa.T) - 1;
          }
          const int s0 = fa.row_start[first[0]], s1 = fa.row_start[first[1]], e0 = fa.row_start[last[0]], e1 = fa.row_start[last[1]];
          it.kv_lo = fa_first_key(first[0], s0, fa.window);
          it.n[0] = fa_num_kv_tiles(it.q0, fa.T, it.kv_lo, KN);
          it.n[1] = fa_num_kv_tiles(it.q0 + kFaM, fa.T, it.kv_lo, KN);
          it.jlo[1] = fa_first_kv_tile(fa_first_key(first[1], s1, fa.window), it.kv_lo, it.n[1], KN);
          it.max_start[0] = fa_first_key(last[0], e0, fa.window);
          it.max_start[1] = fa_first_key(last[1], e1, fa.window);
        }
        if (!mbar_wait(&sh->item_empty[i & 1], ((i >> 1) & 1) ^ 1, abort_flag)) { ok = false; break; }
        sh->item[i & 1] = it;
        mbar_arrive(&sh->item_full[i & 1]);
        if (!it.valid) break;
      }
      if (!ok) {
        sh->abort_flag = 1;
        atomicCAS(err, 0, kFaErrItems);
      }
    }
  } else {
    // ---------------- softmax / correction / epilogue: one group per query tile ----------------
    setmaxnreg_inc<kFaRegsSoftmax>();
    const int t = (warp - 4) >> 2;               // query tile of this group
    const int quad = warp & 3;                   // TMEM lane quadrant this warp may access
    const int r = quad * 32 + lane;
    const uint32_t lane_off = (uint32_t)(quad * 32) << 16;
    const uint32_t t_s = tmem_base + lane_off + t * 128;
    const uint32_t t_o = tmem_base + lane_off + 256 + t * 128;
    const float scale_log2 = fa.scale_log2;
    bool ok = true;
    auto fail = [&]() {
      ok = false;
      sh->abort_flag = 1;
      atomicCAS(err, 0, kFaErrSoftmax);
    };
    int ns = 0, no = 0;                          // score tiles and finished query tiles so far
    for (int i = 0;; ++i) {
      if (!mbar_wait(&sh->item_full[i & 1], (i >> 1) & 1, abort_flag)) fail();
      if (__any_sync(0xffffffffu, !ok)) break;
      const FaItem* it = &sh->item[i & 1];
      const int valid = it->valid, q0 = it->q0, h = it->h, kv_lo = it->kv_lo, jlo = it->jlo[t], my_n = it->n[t];
      const int max_row_start = it->max_start[t];
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh->item_empty[i & 1]);
      if (!valid) break;
      if (my_n <= jlo) continue;
      const int tile_first = q0 + t * kFaM, row = tile_first + r;
      const bool row_valid = row < fa.T;
      const int my_start = row_valid ? fa_first_key(row, fa.row_start[row], fa.window) : 0x7fffffff;
      float m_used = -1e30f, l = 0.f;
      // ALiBi bias in units of the raw score: (slope / scale) * (key - query), so that score * scale_log2 carries it
      const float alibi_s = fa.alibi_slopes != nullptr ? fa.alibi_slopes[h] * 1.4426950408889634f / scale_log2 : 0.f;
      for (int j = jlo; j < my_n; ++j) {
        // this also says that P·V of the step before has been added: it was issued earlier
        if (!mbar_wait(&sh->s_full[t], ns++ & 1, abort_flag)) fail();
        tc_fence_after();
        uint32_t s[KN];
#pragma unroll
        for (int c = 0; c < KN; c += 32) tmem_ld_32x32(t_s + c, s + c);
        tmem_ld_wait();
        const int k0 = kv_lo + j * KN;
        const bool need_mask = fa_tile_needs_mask(k0, tile_first, max_row_start, KN);
        if (need_mask) {
          // 32 keys at a time: those that a row sees are a range of bits, and where that is all of them for all rows of the warp
          // (three of four groups left of a diagonal) nothing is left to do
#pragma unroll
          for (int c = 0; c < KN; c += 32) {
            const int lo = my_start - (k0 + c), hi = row - (k0 + c);
            uint32_t seen = hi < 0 ? 0u : 0xffffffffu >> (31 - min(hi, 31));
            if (lo > 0) seen = lo > 31 ? 0u : seen & (0xffffffffu << lo);
            if (__any_sync(0xffffffffu, seen != 0xffffffffu)) {
#pragma unroll
              for (int i = 0; i < 32; ++i)
                if (!(seen >> i & 1)) s[c + i] = 0xff800000u;   // -inf
            }
          }
        }
        if (fa.alibi_slopes != nullptr) {
          const float d0 = (float)(k0 - row);
#pragma unroll
          for (int i = 0; i < KN; ++i)
            s[i] = __float_as_uint(fmaf(alibi_s, d0 + (float)i, __uint_as_float(s[i])));   // -inf stays -inf
        }
        float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
#pragma unroll
        for (int i = 0; i < KN; i += 8) {
          mx0 = fmax3(mx0, __uint_as_float(s[i]), __uint_as_float(s[i + 1]));
          mx1 = fmax3(mx1, __uint_as_float(s[i + 2]), __uint_as_float(s[i + 3]));
          mx2 = fmax3(mx2, __uint_as_float(s[i + 4]), __uint_as_float(s[i + 5]));
          mx3 = fmax3(mx3, __uint_as_float(s[i + 6]), __uint_as_float(s[i + 7]));
        }
        const float mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3)) * scale_log2;
        const float m_new = fmaxf(m_used, mx);
        const bool grow = (m_new - m_used) > kFaRescaleThreshold;
        float alpha = 1.f;
        if (grow) {
          alpha = exp2f(m_used - m_new);
          m_used = m_new;
          l *= alpha;
        }
        if (j > jlo && __any_sync(0xffffffffu, grow)) {
#pragma unroll 1
          for (int c = 0; c * 32 < dv; ++c) {
            uint32_t v[32];
            tmem_ld_32x32(t_o + c * 32, v);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * alpha);
            tmem_st_32x32(t_o + c * 32, v);
          }
        }
        // P = exp2(s*scale - m_used) as pairs of bf16 over the first columns of the scores, 32 keys at a time; the product with V
        // starts on the first part.  Everything but ex2 and the conversion works on pairs (or takes three operands).
        float2 ps0 = make_float2(0.f, 0.f), ps1 = ps0;
        const float2 scale2 = make_float2(scale_log2, scale_log2), neg_m = make_float2(-m_used, -m_used);
#pragma unroll
        for (int c = 0; c < KN; c += 32) {
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const float2 x = ffma2(make_float2(__uint_as_float(s[c + i]), __uint_as_float(s[c + i + 1])), scale2, neg_m);
            const float p0 = ex2_approx(x.x), p1 = ex2_approx(x.y);
            if (i & 2) ps1 = fadd2(ps1, make_float2(p0, p1));
            else ps0 = fadd2(ps0, make_float2(p0, p1));
            const __nv_bfloat162 b = __floats2bfloat162_rn(p0, p1);
            pk[i >> 1] = *reinterpret_cast<const uint32_t*>(&b);
          }
          tmem_st_32x16(t_s + c / 2, pk);
          if (c + 32 == Cfg::kFirst || c + 32 == KN) {
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(c + 32 == KN ? &sh->p_full[t] : &sh->p_first[t]);
          }
        }
        l += (ps0.x + ps0.y) + (ps1.x + ps1.y);
      }
      // ---------------- epilogue: O / l -> bf16 -> global; LSE ----------------
      if (!mbar_wait(&sh->o_full[t], no++ & 1, abort_flag)) fail();
      tc_fence_after();
      // the sink is one more term of the denominator, without a key or a value
      if (fa.sink != nullptr) l += exp2f(fa.sink[h] * 1.4426950408889634f - m_used);
      float inv_l = row_valid ? 1.f / l : 0.f;
      if (fa.gate != nullptr && row_valid)
        inv_l *= 1.f / (1.f + __expf(-__bfloat162float(fa.gate[(size_t)row * fa.ldg + h])));
      const bool write = row_valid && ok && !*abort_flag;
      // Through the warp's own 32 rows x 64 columns of shared memory and out by the TMA unit, which leaves out what lies past the
      // tensor: a row at a time from registers touches 32 lines a store, 4000 cycles a tile.
      uint8_t* stage = smem + Cfg::kOps + (warp - 4) * 4096;
      const bool out_ok = __all_sync(0xffffffffu, ok && !*abort_flag);
#pragma unroll 1
      for (int c = 0; c < dv; c += 64) {
        uint32_t v[64];
        tmem_ld_32x32(t_o + c, v);
        tmem_ld_32x32(t_o + c + 32, v + 32);
        tmem_ld_wait();
        if (lane == 0) tma_store_wait_read<0>();         // of the chunk, or the item, before
        __syncwarp();
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          float f[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) f[i] = __uint_as_float(v[g * 8 + i]) * inv_l;
          *reinterpret_cast<bf16x8*>(stage + lane * 128 + ((g ^ (lane & 7)) << 4)) = pack8(f);
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && out_ok) {
          tma_store_3d(&tmO, stage, c, h, tile_first + quad * 32);
          tma_store_commit();
        }
      }
      if (write && fa.lse != nullptr) fa.lse[(size_t)h * fa.T + row] = m_used * 0.6931471805599453f + logf(l);
    }
    if (lane == 0) tma_store_wait_read<0>();
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) {
    // error path: give copies / MMAs still in flight time to land before smem and TMEM go away
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

int make_tmap_bf16_heads(CUtensorMap* map, const void* ptr, uint64_t dim, uint64_t heads, uint64_t rows,
                         uint64_t row_stride_bytes, uint32_t box_dim, uint32_t box_rows, uint64_t head_stride_bytes = 0);

template <int KN, int NC>
static int launch_flash_fwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tq2,
                            const CUtensorMap& tk2, const FaArgs& fa, cudaStream_t stream) {
  CUtensorMap to;
  const int rc = make_tmap_bf16_heads(&to, fa.out, fa.dv, fa.Hq, fa.T, (uint64_t)fa.Hq * fa.dv * 2, 64, 32);
  if (rc) return rc;
  auto kern = flash_fwd_kernel<KN, NC>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, FaCfg<KN, NC>::kSmemBytes);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  const long long grid = (long long)((fa.T + 2 * kFaM - 1) / (2 * kFaM)) * fa.Hq;
  if (grid > 0x7fffffff) return -2;
  FaArgs args = fa;
  args.head_group = fa_head_group(fa.T, fa.Hq, fa.Hk, fa.d, fa.dv);
  kern<<<(unsigned)grid, kFaThreads, FaCfg<KN, NC>::kSmemBytes, stream>>>(tq, tk, tv, tq2, tk2, to, args);
  return launch_status();
}

}  // namespace ell

using namespace ell;

// Host-only: the forward kernel's plan for host-resident row_start [T], from the kernel's own arithmetic.  For every
// CTA tile pair p (query rows 256p ..) and tile t in {0, 1}: out[(2p + t) * 3 + {0, 1, 2}] = first key row, number of
// key tiles, and a bit mask (bit j set = key tile j is masked element-wise; only the first 31 tiles are recorded).
ELL_API int ell_flash_fwd_plan(const int* row_start, int T, int* out) {
  const int n_pairs = (T + 2 * kFaM - 1) / (2 * kFaM);
  for (int p = 0; p < n_pairs; ++p) {
    const int q0 = p * 2 * kFaM, kv_lo = row_start[q0];
    for (int t = 0; t < 2; ++t) {
      const int tile_first = q0 + t * kFaM;
      const int n = fa_num_kv_tiles(tile_first, T, kv_lo);
      const int last_row = (tile_first + kFaM < T ? tile_first + kFaM : T) - 1;
      const int max_row_start = n > 0 ? row_start[last_row] : 0;
      int bits = 0;
      for (int j = 0; j < n && j < 31; ++j)
        if (fa_tile_needs_mask(kv_lo + j * kFaN, tile_first, max_row_start)) bits |= 1 << j;
      int* o = out + (2 * p + t) * 3;
      o[0] = kv_lo;
      o[1] = n;
      o[2] = bits;
    }
  }
  return n_pairs;
}

// Host-only: the key tiles, counted from the pair's first, that the second query tile of every pair of 128-row tiles leaves out at the
// start of its walk (all keys of a document, or before a window, that its rows do not see); from the kernel's own arithmetic.
ELL_API int ell_flash_fwd_skipped(const int* row_start, int T, int window, int kn, int* out) {
  const int n_pairs = (T + 2 * kFaM - 1) / (2 * kFaM);
  if (window <= 0) window = 0x7fffffff;
  for (int p = 0; p < n_pairs; ++p) {
    const int q0 = p * 2 * kFaM, q1 = q0 + kFaM < T ? q0 + kFaM : T - 1;
    const int kv_lo = fa_first_key(q0, row_start[q0], window);
    out[p] = fa_first_kv_tile(fa_first_key(q1, row_start[q1], window), kv_lo, fa_num_kv_tiles(q0 + kFaM, T, kv_lo, kn), kn);
  }
  return n_pairs;
}

// q [T, Hq, d], k [T, Hk, d], v [T, Hk, dv] bf16 with row strides (in elements) q_stride / k_stride / v_stride (views
// into the packed QKV GEMM output are fine), d and dv multiples of 8 up to 128; out [T, Hq, dv] contiguous; lse [Hq, T]
// fp32 or null; row_start [T] int32 (document start of every token).  Causal.
// alibi_slopes, sink: fp32 [Hq] or null.  window: keys a row sees at most (<= 0: all of its document before it).
ELL_API int ell_flash_attn_fwd(const void* q, const void* k, const void* v, void* out, float* lse, const int* row_start,
                               int T, int Hq, int Hk, int d, int dv, int q_stride, int k_stride, int v_stride, float scale,
                               const float* alibi_slopes, const float* sink, int window, int* err,
                               cudaStream_t stream) {
  if (T <= 0) return 0;
  if (Hq % Hk || d < 8 || d > kFaD || d % 8 || dv < 8 || dv > kFaD || dv % 8) return -2;
  CUtensorMap tq, tk, tv;
  int rc = make_tmap_bf16_heads(&tq, q, d, Hq, T, (uint64_t)q_stride * 2, 64, 128);
  if (rc) return rc;
  rc = make_tmap_bf16_heads(&tk, k, d, Hk, T, (uint64_t)k_stride * 2, 64, 128);
  if (rc) return rc;
  rc = make_tmap_bf16_heads(&tv, v, dv, Hk, T, (uint64_t)v_stride * 2, 64, 128);
  if (rc) return rc;
  FaArgs fa{(__nv_bfloat16*)out, lse, row_start, T, Hq, Hk, d, 0, dv, window > 0 ? window : 0x7fffffff,
            scale * 1.4426950408889634f, alibi_slopes, sink, nullptr, 0, err};
  return launch_flash_fwd<kFaN, 2>(tq, tk, tv, tq, tk, fa, stream);
}

// Latent attention on packed prompts: q [T, H, d + d2] (rows of q_stride), k [T, H, d] the heads' own key parts, k2 [T, d2]
// the part they share, v [T, H, dv], all bf16 with row strides in elements; sizes are multiples of 8, d and d2 take at
// most three 64-column chunks together, dv at most 128.  window <= 0: none.  gate: [T, H] rows of ldg, or null.
ELL_API int ell_flash_attn_latent(const void* q, const void* k, const void* k2, const void* v, void* out,
                                  const int* row_start, const void* gate, int T, int H, int d, int d2, int dv, int q_stride,
                                  int k_stride, int k2_stride, int v_stride, int ldg, int window, float scale, int* err,
                                  cudaStream_t stream) {
  if (T <= 0) return 0;
  const int chunks = (d + 63) / 64 + (d2 + 63) / 64;
  if (d < 8 || d % 8 || d2 < 8 || d2 % 8 || chunks > 3 || dv < 8 || dv > kFaD || dv % 8) return -2;
  const int kn = chunks > 2 ? 64 : 128;
  const uint64_t head = (uint64_t)(d + d2) * 2;
  CUtensorMap tq, tq2, tk, tk2, tv;
  int rc = make_tmap_bf16_heads(&tq, q, d, H, T, (uint64_t)q_stride * 2, 64, 128, head);
  if (!rc) rc = make_tmap_bf16_heads(&tq2, (const __nv_bfloat16*)q + d, d2, H, T, (uint64_t)q_stride * 2, 64, 128, head);
  if (!rc) rc = make_tmap_bf16_heads(&tk, k, d, H, T, (uint64_t)k_stride * 2, 64, kn);
  if (!rc) rc = make_tmap_bf16_heads(&tk2, k2, d2, 1, T, (uint64_t)k2_stride * 2, 64, kn);
  if (!rc) rc = make_tmap_bf16_heads(&tv, v, dv, H, T, (uint64_t)v_stride * 2, 64, kn);
  if (rc) return rc;
  FaArgs fa{(__nv_bfloat16*)out, nullptr, row_start, T, H, H, d, d2, dv, window > 0 ? window : 0x7fffffff,
            scale * 1.4426950408889634f, nullptr, nullptr, (const __nv_bfloat16*)gate, ldg, err};
  if (kn == 64) return launch_flash_fwd<64, 3>(tq, tk, tv, tq2, tk2, fa, stream);
  return launch_flash_fwd<128, 2>(tq, tk, tv, tq2, tk2, fa, stream);
}
