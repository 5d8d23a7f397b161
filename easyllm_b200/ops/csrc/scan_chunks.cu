// The scans of recurrent.cu for prompts: 16 tokens at a time instead of one.
//
// Token by token a scan of a long sequence is a chain of reductions, 0.13 us (time mixing) to 0.26 us (delta rule) a token however
// idle the GPU is.  Over a chunk of 16 tokens with the state S0 in front of it, and P_i the product of the chunk's decays up to
// token i (delta rule: with token i's own; time mixing: without, its output is read before the decay),
//   delta rule    (I + diag(beta) tril(A^kk, -1)) E = diag(beta) (V - (K o P) S0),   O = (Q o P) S0 + tril(A^qk) E
//   time mixing   E = V,                                                             O = (R o P) S0 + tril(A^rk) V
//   both          S = P_16 o S0 + (K o P_16 / P_i)^T E
// with A_ij = sum_c x_ic k_jc prod(decays between j and i).  No decay is divided by: a product between j and i is the product from
// a point between them up to i times the one from j up to that point (points at 8, then 4 and 12, ...), and P_16 / P_i is a product
// from the end, so decays of any size, zeros too, give what the recurrence gives.
//
// chunk_prepare_kernel, one CTA per (chunk, head), all at once: the scaled rows, A, and the inverse of the triangular matrix, as
// one fp32 record per chunk.  chunk_scan_kernel, one CTA per (16 value columns, head, sequence), walks the chunks: a loader warp
// brings records (one bulk copy each) and the values into a ring; the other warps hold 16 key rows of the state each, in the layout of
// mma.sync's accumulators, which is also that of its left operand.
//
// Precision: fp32 or better throughout.  Products of decays are pairs of floats, sums over the channels are added up in 64 bits.  The
// products with the state take both operands as three bf16 parts (24 bits) and sum six of the nine partial products in fp32; the
// state itself is updated by fused multiply-adds.  Against 64 bits, relative errors of 700 tokens of 128 x 128 heads are 0.94e-7 (time
// mixing; token by token 1.00e-7) and 1.04e-7 (delta rule; 1.22e-7), of 2500 tokens with decays near 1 1.5e-7 (2.8e-7) and 1.5e-7
// (3.1e-7): fewer steps are rounded.  With products and sums in one float they were 1.21e-7 and 1.42e-7 for 700 tokens, larger than
// token by token.  (With fp32 multiply-adds in place of the bf16 parts: the same errors and 450 us where the delta rule takes 370,
// since the sums over key rows then cross the lanes of a warp.)
//
// Bound by the issue of some 550 instructions a warp and chunk (delta rule; half of the slots are used, the rest waits on the chain
// from the state to the next one).  One sequence of 4096 tokens, both launches: 16 heads of 128 x 128, delta rule, 1044 -> 430 us; 32
// heads of 64 x 64, time mixing, 516 -> 265.  8 sequences of 512: 530 -> 397 and 207 -> 168.
#include "sm100.cuh"
#include "vec.cuh"

namespace ell {
using sm100::bulk_load;
using sm100::fence_barrier_init;
using sm100::mbar_arrive;
using sm100::mbar_expect_tx;
using sm100::mbar_init;
using sm100::mbar_wait;

constexpr int kCk = 16;                    // tokens of a chunk
constexpr int kCkCols = 16;                // value columns of a CTA
constexpr int kCkMat = 20;                 // row stride of the 16 x 16 matrices
constexpr int kCkCol = 24;                 // stride of a column's 16 tokens
constexpr int kCkStages = 4;
constexpr int kErrScan = 41;

enum ScanMode { kWkv = 0, kDelta = 1 };

// Record of a chunk in floats: scaled rows (delta: of q and of k; time mixing: of r) | scaled keys | decay of the chunk | A | inverse.
template <int MODE, int DP>
struct Rec {
  static constexpr int kRows = (MODE == kDelta ? 2 : 1) * kCk;
  static constexpr int kStride = DP + 8;             // of the scaled rows: a fragment's 4 x 8 words lie in 32 banks
  static constexpr int kQ = 0, kK = kCk * kStride, kS = kRows * kStride, kP = kS + kCk * kStride, kA = kP + DP;
  static constexpr int kT = kA + kCk * kCkMat;
  static constexpr int kFloats = kT + (MODE == kDelta ? kCk * kCkMat : 0);
};

struct ChunkArgs {
  const void *q, *k, *v;        // delta: fp32; wkv: activation type.  q is r in wkv
  const float *g, *beta, *u;
  float* o;
  float* state;                 // [slots, H, dv, dp] or null
  const int *cu, *slots, *pos0;
  float* rec;
  float* carry;                 // [n_seq, H, dv, DP]: the state between two launches over one sequence, or null
  int H, G, d, dv, ldq, ldk, ldv, n_seq;
  int c0, c1, per_seq;          // chunks of this launch; records per sequence (0: counted by tokens)
  int final;                    // no chunks come after this launch
  int* err;
};

// First record of a sequence.  Sequences of n tokens have at most n / 16 + 1 chunks.
__device__ __forceinline__ size_t first_record(const ChunkArgs& a, int s, int start) {
  return a.per_seq > 0 ? (size_t)s * a.per_seq : (size_t)(start / kCk + s);
}

// Product of up to 16 decays as an unevaluated sum of two floats: in one float its rounding errors, one a factor, were most of the
// error of a chunk.
struct DecayProduct {
  float hi = 1.f, lo = 0.f;
  __device__ __forceinline__ void times(float g) {
    const float h = __fmul_rn(hi, g);
    lo = fmaf(lo, g, fmaf(hi, g, -h));
    hi = h;
  }
  __device__ __forceinline__ float of(float x) const { return fmaf(x, hi, __fmul_rn(x, lo)); }
};

__device__ __forceinline__ double dot4(const float* x, const float* y) {
  const float4 a = *reinterpret_cast<const float4*>(x), b = *reinterpret_cast<const float4*>(y);
  return (double)fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, a.x * b.x)));
}

// Dot products of one level: token i of a right half with token j of the left half before it, for halves of HS tokens.  A thread
// takes a share of the channels of one pair; neighbours add theirs.
template <int MODE, int HS, int DP>
__device__ __forceinline__ void level_products(const float* rows, const float* keys, float* aqk, float* akk) {
  constexpr int kStride = DP + 4, kPairs = 8 * HS, kDots = kPairs * (MODE == kDelta ? 2 : 1), kShares = kDots < DP ? DP / kDots : 1;
#pragma unroll
  for (int first = 0; first < kDots; first += DP / kShares) {
    const int dot = first + threadIdx.x / kShares, share = threadIdx.x % kShares;
    const int pair = dot % kPairs, block = pair / (HS * HS), in = pair % (HS * HS);
    const int i = block * 2 * HS + HS + in / HS, j = block * 2 * HS + in % HS;
    const bool kk = MODE == kDelta && dot >= kPairs;
    const float* x = (kk ? keys : rows) + i * kStride;
    const float* y = keys + j * kStride;
    double sum = 0.;
#pragma unroll 8
    for (int c = share * 4; c < DP; c += kShares * 4) sum += dot4(x + c, y + c);
#pragma unroll
    for (int o = kShares / 2; o >= 1; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (share == 0) (kk ? akk : aqk)[i * kCkMat + j] = (float)sum;
  }
}

// One level: the rows of its right halves scaled by the decays from the middle on, the keys of its left halves by those up to it.
template <int MODE, int HS, int DP>
__device__ __forceinline__ void level(const float (&q)[kCk], const float (&k)[kCk], const float (&g)[kCk], float* rows, float* keys,
                                      float* aqk, float* akk) {
  constexpr int kStride = DP + 4;
  const int c = threadIdx.x;
#pragma unroll
  for (int mid = HS; mid < kCk; mid += 2 * HS) {
    DecayProduct p, back;
#pragma unroll
    for (int i = mid; i < mid + HS; ++i) {
      if (MODE == kDelta) p.times(g[i]);
      rows[i * kStride + c] = p.of(q[i]);
      if (MODE == kDelta) keys[i * kStride + c] = p.of(k[i]);
      if (MODE == kWkv) p.times(g[i]);
    }
#pragma unroll
    for (int j = mid - 1; j >= mid - HS; --j) {
      keys[j * kStride + c] = back.of(k[j]);
      back.times(g[j]);
    }
  }
  __syncthreads();
  level_products<MODE, HS, DP>(rows, keys, aqk, akk);
  __syncthreads();
}

// One thread per channel.
template <int MODE, typename T, int DP>
__global__ void __launch_bounds__(DP) chunk_prepare_kernel(const ChunkArgs a) {
  using R = Rec<MODE, DP>;
  constexpr int kStride = DP + 4;
  __shared__ float4 rows4[kCk * kStride / 4], keys4[kCk * kStride / 4];
  __shared__ float aqk[kCk * kCkMat], akk[kCk * kCkMat], beta[kCk];
  float *rows = reinterpret_cast<float*>(rows4), *keys = reinterpret_cast<float*>(keys4);
  // one CTA a record: chunks of this round by sequence, or, counted by tokens, the sequence whose records these are
  int s = blockIdx.z, chunk = a.c0 + blockIdx.x;
  const int h = blockIdx.y;
  if (a.per_seq == 0) {
    int past = a.n_seq;
    while (past - s > 1) {
      const int mid = (s + past) / 2;
      if (first_record(a, mid, a.cu[mid]) <= blockIdx.x) s = mid;
      else past = mid;
    }
    chunk = blockIdx.x - (int)first_record(a, s, a.cu[s]);
  }
  const int start = a.cu[s], n_tok = a.cu[s + 1] - start, t0 = chunk * kCk;
  if (chunk < 0 || t0 >= n_tok) return;
  const int cnt = min(kCk, n_tok - t0), c = threadIdx.x, hk = h / (a.H / a.G);
  float* rec = a.rec + ((first_record(a, s, start) + (a.per_seq > 0 ? blockIdx.x : chunk)) * a.H + h) * R::kFloats;
  float q[kCk], k[kCk], g[kCk];
  const bool in = c < a.d;
  const size_t first = (size_t)start + t0;
  const T* qp = reinterpret_cast<const T*>(a.q) + first * a.ldq + (size_t)hk * a.d + c;
  const T* kp = reinterpret_cast<const T*>(a.k) + first * a.ldk + (size_t)hk * a.d + c;
  const float* gp = a.g + (first * a.H + h) * a.d + c;
#pragma unroll
  for (int i = 0; i < kCk; ++i) {
    const bool there = in && i < cnt;
    q[i] = there ? to_f<T>(qp[0]) : 0.f;
    k[i] = there ? to_f<T>(kp[0]) : 0.f;
    g[i] = there ? gp[0] : 1.f;
    qp += a.ldq;
    kp += a.ldk;
    gp += a.H * a.d;
  }
  for (int i = threadIdx.x; i < kCk * kCkMat; i += DP) aqk[i] = akk[i] = 0.f;
  if (MODE == kDelta && threadIdx.x < kCk)
    beta[threadIdx.x] = threadIdx.x < cnt ? a.beta[(first + threadIdx.x) * a.H + h] : 0.f;
  {
    DecayProduct p, back;
#pragma unroll
    for (int i = 0; i < kCk; ++i) {
      if (MODE == kDelta) p.times(g[i]);
      rec[R::kQ + i * R::kStride + c] = p.of(q[i]);
      if (MODE == kDelta) rec[R::kK + i * R::kStride + c] = p.of(k[i]);
      if (MODE == kWkv) p.times(g[i]);
    }
    rec[R::kP + c] = p.hi + p.lo;
#pragma unroll
    for (int i = kCk - 1; i >= 0; --i) {
      rec[R::kS + i * R::kStride + c] = back.of(k[i]);
      back.times(g[i]);
    }
    // the diagonal of A: q . k, or the bonus of the token itself
    const float u = MODE == kWkv && in ? a.u[(size_t)h * a.d + c] : 1.f;
#pragma unroll
    for (int i = 0; i < kCk; ++i) {
      rows[i * kStride + c] = q[i] * u;
      keys[i * kStride + c] = k[i];
    }
  }
  __syncthreads();
  {
    constexpr int kShares = DP / kCk;
    const int i = threadIdx.x / kShares, share = threadIdx.x % kShares;
    double sum = 0.;
#pragma unroll
    for (int x = share * 4; x < DP; x += kShares * 4) sum += dot4(rows + i * kStride + x, keys + i * kStride + x);
#pragma unroll
    for (int o = kShares / 2; o >= 1; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (share == 0) aqk[i * kCkMat + i] = (float)sum;
  }
  __syncthreads();
  level<MODE, 8, DP>(q, k, g, rows, keys, aqk, akk);
  level<MODE, 4, DP>(q, k, g, rows, keys, aqk, akk);
  level<MODE, 2, DP>(q, k, g, rows, keys, aqk, akk);
  level<MODE, 1, DP>(q, k, g, rows, keys, aqk, akk);
  for (int i = threadIdx.x; i < kCk * kCkMat; i += DP) rec[R::kA + i] = aqk[i];
  if (MODE == kDelta && threadIdx.x < kCk) {
    // column `threadIdx.x` of (I + diag(beta) tril(A^kk, -1))^-1 diag(beta), by forward substitution
    float x[kCk];
#pragma unroll
    for (int i = 0; i < kCk; ++i) {
      float e = i == (int)threadIdx.x ? 1.f : 0.f;
#pragma unroll
      for (int j = 0; j < i; ++j) e = fmaf(-akk[i * kCkMat + j], x[j], e);
      x[i] = i < (int)threadIdx.x ? 0.f : beta[i] * e;
      rec[R::kT + i * kCkMat + threadIdx.x] = x[i];
    }
  }
}

// ---- the walk over the chunks ----
// Warp w holds key rows 16 w .. 16 w + 15 of the 16 columns.
template <int MODE, int DP>
struct ScanSmem {
  static constexpr int kWarps = DP / 16, kColsOfWarp = kCkCols / kWarps;           // columns a warp finishes
  static constexpr int kThreads = (kWarps + 1) * 32;                               // and the loader
  static constexpr int kStageFloats = Rec<MODE, DP>::kFloats + kCkCols * kCkCol;   // record | values [column][token]
  static constexpr int kPart = Rec<MODE, DP>::kRows * kCkMat;                      // a warp's share of the sums: [row][column]
  static constexpr int kFloats = kCkStages * kStageFloats + 2 * kWarps * kPart + 2 * kCkCols * kCkCol;   // and V - X, E
  static constexpr int kBytes = kFloats * 4;
};

// x, y as three bf16 parts each: 24 bits, nothing is lost.
struct Parts {
  uint32_t p[3];
};
__device__ __forceinline__ Parts split3(float x, float y) {
  Parts r;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    __nv_bfloat162 b = __floats2bfloat162_rn(x, y);
    r.p[i] = *reinterpret_cast<uint32_t*>(&b);
    x -= __uint_as_float(r.p[i] << 16);
    y -= __uint_as_float(r.p[i] & 0xffff0000u);
  }
  return r;
}
__device__ __forceinline__ void mma_parts(float* c, const uint32_t a0, const uint32_t a1, const uint32_t a2, const uint32_t a3,
                                          const uint32_t b0, const uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// acc[x] = a b[x] over 16 k in fp32: the products of parts down to 2^-16 of the largest, the small ones summed apart.  The
// products of one tile wait for one another (35 cycles each), so the tiles are interleaved.
template <int TILES>
__device__ __forceinline__ void mma_f32(float (&acc)[TILES][4], const Parts (&a)[4], const Parts (&b)[TILES][2]) {
  constexpr int order[6][2] = {{0, 2}, {0, 1}, {2, 0}, {1, 0}, {1, 1}, {0, 0}};
  float small[TILES][4];
#pragma unroll
  for (int x = 0; x < TILES; ++x)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[x][i] = small[x][i] = 0.f;
#pragma unroll
  for (int i = 0; i < 6; ++i)
#pragma unroll
    for (int x = 0; x < TILES; ++x) {
      const int u = order[i][0], v = order[i][1];
      mma_parts(i & 1 ? acc[x] : small[x], a[0].p[u], a[1].p[u], a[2].p[u], a[3].p[u], b[x][0].p[v], b[x][1].p[v]);
    }
#pragma unroll
  for (int x = 0; x < TILES; ++x)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[x][i] += small[x][i];
}

// Barrier of the warps that hold the state; tells all of them whether any has given up.
template <int THREADS>
__device__ __forceinline__ bool any_failed(bool failed) {
  uint32_t any;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
      "bar.red.or.pred p, 1, %2, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(any) : "r"((uint32_t)failed), "n"(THREADS) : "memory");
  return any != 0;
}
template <int THREADS>
__device__ __forceinline__ void state_barrier() {
  asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory");
}

// Half a token's values of this CTA's columns (8 of 16) as they lie in memory, zeros where there are none: a load is not waited
// for before its stage is free.
template <typename T>
struct RawValues {
  uint4 r[sizeof(T) / 2];
};
template <typename T>
__device__ __forceinline__ RawValues<T> load_values(const ChunkArgs& a, int start, int t, int n_tok, int h, int col) {
  RawValues<T> x;
  const bool in = t < n_tok && col < a.dv;
  const uint4* p = reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(a.v) + (size_t)(start + t) * a.ldv + (size_t)h * a.dv + col);
#pragma unroll
  for (int i = 0; i < (int)sizeof(T) / 2; ++i) x.r[i] = in ? p[i] : make_uint4(0, 0, 0, 0);
  return x;
}

// Tokens t0 .. t1 - 1 of a sequence one by one, as scan_kernel computes them, for a warp's NC columns from `col` on.  Lane l holds
// key rows l, l + 32, ... of them.  What chunks cannot do comes here: it is slow (0.5 us a token) and rare.  mend: only outputs
// that are not finite are written.
__device__ __forceinline__ bool is_finite(float x) { return x * 0.f == 0.f; }
template <int MODE, typename T, int DP, int NC>
__device__ __noinline__ void walk_tokens(const ChunkArgs& a, int start, int t0, int t1, int h, int col, float (&S)[NC][DP / 32],
                                         bool mend) {
  constexpr int J = DP / 32;
  const int lane = threadIdx.x & 31, hk = h / (a.H / a.G);
  float u[J];
#pragma unroll
  for (int j = 0; j < J; ++j) u[j] = MODE == kWkv && lane + 32 * j < a.d ? a.u[(size_t)h * a.d + lane + 32 * j] : 0.f;
  for (int t = t0; t < t1; ++t) {
    const size_t at = (size_t)start + t;
    float q[J], k[J], g[J], dot = 0.f;
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const int r = lane + 32 * j;
      const bool in = r < a.d;
      q[j] = in ? to_f<T>(reinterpret_cast<const T*>(a.q)[at * a.ldq + (size_t)hk * a.d + r]) : 0.f;
      k[j] = in ? to_f<T>(reinterpret_cast<const T*>(a.k)[at * a.ldk + (size_t)hk * a.d + r]) : 0.f;
      g[j] = in ? a.g[(at * a.H + h) * a.d + r] : 0.f;
      dot = MODE == kWkv ? fmaf(q[j] * k[j], u[j], dot) : fmaf(q[j], k[j], dot);
    }
    dot = warp_sum(dot);
    const float beta = MODE == kDelta ? a.beta[at * a.H + h] : 0.f;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      if (col + c >= a.dv) break;                      // the same in all lanes
      const float v = to_f<T>(reinterpret_cast<const T*>(a.v)[at * a.ldv + (size_t)h * a.dv + col + c]);
      float ks = 0.f, qs = 0.f;
#pragma unroll
      for (int j = 0; j < J; ++j) {
        if (MODE == kDelta) {
          S[c][j] *= g[j];
          ks = fmaf(k[j], S[c][j], ks);
        }
        qs = fmaf(q[j], S[c][j], qs);
      }
      if (MODE == kDelta) ks = warp_sum(ks);
      qs = warp_sum(qs);
      const float e = MODE == kDelta ? beta * (v - ks) : v;
#pragma unroll
      for (int j = 0; j < J; ++j)
        if (lane + 32 * j < a.d) S[c][j] = MODE == kDelta ? fmaf(k[j], e, S[c][j]) : fmaf(g[j], S[c][j], k[j] * e);
      float* o = a.o + (at * a.H + h) * a.dv + col + c;
      if (lane == 0 && !(mend && is_finite(*o))) *o = fmaf(dot, e, qs);
    }
  }
}

template <int MODE, typename T, int DP>
__global__ void __launch_bounds__(ScanSmem<MODE, DP>::kThreads) chunk_scan_kernel(const __grid_constant__ ChunkArgs a) {
  using R = Rec<MODE, DP>;
  using Sm = ScanSmem<MODE, DP>;
  constexpr int kWarps = Sm::kWarps, CW = Sm::kColsOfWarp, kTiles = R::kRows / 8;
  extern __shared__ __align__(128) float sm[];
  __shared__ uint64_t full[kCkStages], empty[kCkStages];
  __shared__ int gave_up;
  __shared__ uint32_t odd_columns;                     // those with values that are not finite
  const int s = blockIdx.z, h = blockIdx.y, col0 = blockIdx.x * kCkCols;
  const int start = a.cu[s], n_tok = a.cu[s + 1] - start;
  const int chunks = (n_tok + kCk - 1) / kCk, last = min(a.c1, chunks), n = last - a.c0;
  if (n <= 0) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kCkStages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], kWarps);
    }
    gave_up = 0;
    odd_columns = 0;
    fence_barrier_init();
  }
  __syncthreads();
  volatile int* stop = &gave_up;

  if (warp == kWarps) {
    const float* rec = a.rec + ((first_record(a, s, start) + (a.per_seq > 0 ? 0 : a.c0)) * a.H + h) * R::kFloats;
    const size_t step = (size_t)a.H * R::kFloats;
    const int tok = lane >> 1, half = (lane & 1) * 8;
    RawValues<T> raw[kCkStages];                       // a round of stages ahead, so that the loads' latency is not on the chain
#pragma unroll
    for (int i = 0; i < kCkStages; ++i) raw[i] = load_values<T>(a, start, (a.c0 + i) * kCk + tok, n_tok, h, col0 + half);
    bool ok = true;
    for (int c = 0; c < n && ok; c += kCkStages) {
#pragma unroll
      for (int i = 0; i < kCkStages; ++i) {
        if (c + i < n && ok) {
          float* st = sm + i * Sm::kStageFloats;
          ok = __all_sync(0xffffffffu, mbar_wait(&empty[i], ((c / kCkStages) & 1) ^ 1, stop));
          if (ok) {
            float v[8];
            load_v<8>(reinterpret_cast<const T*>(raw[i].r), v);
#pragma unroll
            for (int j = 0; j < 8; ++j) st[R::kFloats + (half + j) * kCkCol + tok] = v[j];
            __syncwarp();
            if (lane == 0) {
              mbar_expect_tx(&full[i], R::kFloats * 4);
              bulk_load(st, rec + (size_t)(c + i) * step, R::kFloats * 4, &full[i]);
            }
            raw[i] = load_values<T>(a, start, (a.c0 + c + i + kCkStages) * kCk + tok, n_tok, h, col0 + half);
          }
        }
      }
    }
    if (!ok && lane == 0) {
      *stop = 1;
      atomicCAS(a.err, 0, kErrScan);
    }
  } else {
    // fragments: columns g and g + 8, key rows (or tokens) 2 t, 2 t + 1 of each group of 8
    const int g = lane >> 2, t2 = (lane & 3) * 2, row0 = warp * 16;
    // finished by this lane: token `tok` of columns fin + 2 u
    const int tok = lane >> 1, fin = warp * CW + (lane & 1);
    float* part = sm + kCkStages * Sm::kStageFloats;
    float* rb = part + 2 * kWarps * Sm::kPart;         // V - X, [column][token]
    float* eb = rb + kCkCols * kCkCol;                 // E
    const int sp = (a.d + 31) / 32 * 32;
    // S[j]: key rows row0 + 8 j + t2, + 1 of column g, then of column g + 8
    float S[2][4];
    const int slot = a.state != nullptr ? a.slots[s] : 0;
    const bool kept = a.state != nullptr && a.pos0[s] > 0;
    auto state_at = [&](int c, int r) { return a.state + (((size_t)slot * a.H + h) * a.dv + c) * sp + r; };
    auto carry_at = [&](int c, int r) { return a.carry + (((size_t)s * a.H + h) * a.dv + c) * DP + r; };
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int c = col0 + g + 8 * u, r = row0 + 8 * j + t2;
        const float* from = nullptr;
        if (c < a.dv) from = a.c0 > 0 ? carry_at(c, r) : (kept && r < sp ? state_at(c, r) : nullptr);
        const float2 x = from != nullptr ? *reinterpret_cast<const float2*>(from) : make_float2(0.f, 0.f);
        S[j][2 * u] = x.x;
        S[j][2 * u + 1] = x.y;
      }
    float* o = a.o + ((size_t)(start + a.c0 * kCk + tok) * a.H + h) * a.dv + col0 + fin;
    const size_t o_chunk = (size_t)kCk * a.H * a.dv;
    float probe[CW / 2];                               // becomes NaN with the first output that is not finite
#pragma unroll
    for (int u = 0; u < CW / 2; ++u) probe[u] = 0.f;
    bool failed = false;
    for (int c = 0; c < n; ++c, o += o_chunk) {
      const int i = c % kCkStages;
      failed = !__all_sync(0xffffffffu, mbar_wait(&full[i], (c / kCkStages) & 1, stop));
      const float* st = sm + i * Sm::kStageFloats;
      // this warp's share of the scaled rows' products with the state
      float* mine = part + ((c & 1) * kWarps + warp) * Sm::kPart;
      {
        Parts sa[4], b[kTiles][2];
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int u = 0; u < 2; ++u) sa[2 * j + u] = split3(S[j][2 * u], S[j][2 * u + 1]);
#pragma unroll
        for (int x = 0; x < kTiles; ++x) {
          const float* src = st + (x * 8 + g) * R::kStride + row0 + t2;
          const float2 lo = *reinterpret_cast<const float2*>(src), hi = *reinterpret_cast<const float2*>(src + 8);
          b[x][0] = split3(lo.x, lo.y);
          b[x][1] = split3(hi.x, hi.y);
        }
        float acc[kTiles][4];
        mma_f32<kTiles>(acc, sa, b);
#pragma unroll
        for (int x = 0; x < kTiles; ++x) {
          float* dst = mine + (x * 8 + t2) * kCkMat + g;
          dst[0] = acc[x][0];
          dst[kCkMat] = acc[x][1];
          dst[8] = acc[x][2];
          dst[kCkMat + 8] = acc[x][3];
        }
      }
      failed = any_failed<kWarps * 32>(failed);
      if (failed) break;                               // all of them
      const float* all = part + (c & 1) * kWarps * Sm::kPart;
      auto total = [&](int row, int col) -> float {
        float x[kWarps];
#pragma unroll
        for (int w = 0; w < kWarps; ++w) x[w] = all[w * Sm::kPart + row * kCkMat + col];
#pragma unroll
        for (int m = kWarps / 2; m >= 1; m >>= 1)
#pragma unroll
          for (int w = 0; w < m; ++w) x[w] += x[w + m];
        return x[0];
      };
      // sum over the tokens up to this lane's; later tokens don't touch it (their values may be anything)
      auto causal = [&](float y, const float* matrix, const float* x) -> float {
        float y1 = 0.f;
#pragma unroll
        for (int t = 0; t < kCk; t += 4) {
          float m[4], z[4];
          load_v<4>(matrix + tok * kCkMat + t, m);
          load_v<4>(x + t, z);
          y = fmaf(m[0], t <= tok ? z[0] : 0.f, y);
          y1 = fmaf(m[1], t + 1 <= tok ? z[1] : 0.f, y1);
          y = fmaf(m[2], t + 2 <= tok ? z[2] : 0.f, y);
          y1 = fmaf(m[3], t + 3 <= tok ? z[3] : 0.f, y1);
        }
        return y + y1;
      };
      const float* e = st + R::kFloats;                // E, [column][token]: the values, or
      if (MODE == kDelta) {
#pragma unroll
        for (int u = 0; u < CW; u += 2) rb[(fin + u) * kCkCol + tok] = e[(fin + u) * kCkCol + tok] - total(kCk + tok, fin + u);
        __syncwarp();
#pragma unroll
        for (int u = 0; u < CW; u += 2) eb[(fin + u) * kCkCol + tok] = causal(0.f, st + R::kT, rb + (fin + u) * kCkCol);
        e = eb;
        state_barrier<kWarps * 32>();
      }
      // the state behind the chunk
      {
        Parts ea[4], b[2][2];
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const float2 x = *reinterpret_cast<const float2*>(e + (g + 8 * u) * kCkCol + 8 * j + t2);
            ea[2 * j + u] = split3(x.x, x.y);
          }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float* src = st + R::kS + t2 * R::kStride + row0 + 8 * j + g;
          b[j][0] = split3(src[0], src[R::kStride]);
          b[j][1] = split3(src[8 * R::kStride], src[9 * R::kStride]);
        }
        float acc[2][4];
        mma_f32<2>(acc, ea, b);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float2 p = *reinterpret_cast<const float2*>(st + R::kP + row0 + 8 * j + t2);
          S[j][0] = fmaf(S[j][0], p.x, acc[j][0]);
          S[j][1] = fmaf(S[j][1], p.y, acc[j][1]);
          S[j][2] = fmaf(S[j][2], p.x, acc[j][2]);
          S[j][3] = fmaf(S[j][3], p.y, acc[j][3]);
        }
      }
      // outputs
      float y[CW / 2];
#pragma unroll
      for (int u = 0; u < CW; u += 2) y[u / 2] = causal(total(tok, fin + u), st + R::kA, e + (fin + u) * kCkCol);
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[i]);
#pragma unroll
      for (int u = 0; u < CW; u += 2) {
        probe[u / 2] = fmaf(y[u / 2], 0.f, probe[u / 2]);
        if (col0 + fin + u < a.dv && (a.c0 + c) * kCk + tok < n_tok) o[u] = y[u / 2];
      }
    }
    // where the state of column c goes: to the next launch, or the slot
    auto kept_at = [&](int c, int r) -> float* {
      if (c >= a.dv) return nullptr;
      if (last < chunks && !a.final) return carry_at(c, r);
      return a.state != nullptr && r < sp ? state_at(c, r) : nullptr;
    };
#pragma unroll
    for (int u = 0; u < CW; u += 2)
      if (!is_finite(probe[u / 2])) atomicOr(&odd_columns, 1u << (fin + u));
#pragma unroll
    for (int u = 0; u < 2; ++u)
      if (!is_finite(fmaf(S[0][2 * u], 0.f, S[0][2 * u + 1] * 0.f) + fmaf(S[1][2 * u], 0.f, S[1][2 * u + 1] * 0.f)))
        atomicOr(&odd_columns, 1u << (g + 8 * u));
    state_barrier<kWarps * 32>();
    const uint32_t odd = odd_columns;
    if (failed) {
      *stop = 1;
      if (lane == 0) atomicCAS(a.err, 0, kErrScan);
    } else if (odd != 0 || (last < chunks && a.final)) {
      // The parts of an infinity are not a number, and sums over a chunk may overflow where those over a token do not: what came out
      // not finite is computed again, token by token.  And the other tokens of a sequence longer than the bound that the launches
      // were sized by.
      constexpr int J = DP / 32;
      float* fin = part;                               // [column][row]: the state, by columns
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int u = 0; u < 2; ++u)
          *reinterpret_cast<float2*>(fin + (g + 8 * u) * DP + row0 + 8 * j + t2) = make_float2(S[j][2 * u], S[j][2 * u + 1]);
      state_barrier<kWarps * 32>();
      const int mine = warp * CW;
      float W[CW][J];
      if (odd >> mine & ((1u << CW) - 1)) {
        for (int x = 0; x < CW; ++x)
          for (int j = 0; j < J; ++j) {
            const int c = col0 + mine + x, r = lane + 32 * j;
            W[x][j] = c >= a.dv ? 0.f : (a.c0 > 0 ? *carry_at(c, r) : (kept && r < sp ? *state_at(c, r) : 0.f));
          }
        __syncwarp();                                  // the outputs of this warp's other lanes
        walk_tokens<MODE, T, DP, CW>(a, start, a.c0 * kCk, min(last * kCk, n_tok), h, col0 + mine, W, true);
      }
      for (int x = 0; x < CW; ++x)
        for (int j = 0; j < J; ++j) {
          const float y = fin[(mine + x) * DP + lane + 32 * j];
          if (!(odd >> (mine + x) & 1) || is_finite(y)) W[x][j] = y;
        }
      if (last < chunks && a.final) walk_tokens<MODE, T, DP, CW>(a, start, last * kCk, n_tok, h, col0 + mine, W, false);
      for (int x = 0; x < CW; ++x)
        for (int j = 0; j < J; ++j)
          if (float* to = kept_at(col0 + mine + x, lane + 32 * j)) *to = W[x][j];
    } else {
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int u = 0; u < 2; ++u)
          if (float* to = kept_at(col0 + g + 8 * u, row0 + 8 * j + t2))
            *reinterpret_cast<float2*>(to) = make_float2(S[j][2 * u], S[j][2 * u + 1]);
    }
  }
  __syncthreads();
  if (*stop && threadIdx.x == 0) {                     // copies in flight land before the CTA's memory goes away
    const unsigned long long t0 = sm100::globaltimer_ns();
    while (sm100::globaltimer_ns() - t0 < 200000ull) {
    }
  }
  __syncthreads();
}

// ---- plan of a call ----
// Shorter sequences stay token by token: two launches and their records cost what that many tokens take there (one sequence, us, in
// chunks | by token: time mixing, 128 tokens 30 | 22, 256 tokens 32 | 39; delta rule, 64 tokens 25 | 22, 128 tokens 27 | 39).  The
// records of a call and what is carried between rounds may take kCkMaxBytes; calls that need more go in several rounds over as many
// chunks as fit, with the state carried between them, or token by token where a round would be under kCkMinRound chunks (many
// sequences, which fill the GPU that way too).
//
// Many short sequences beside a long one: the start of a CTA costs more here than token by token, a chunk costs less than 16 tokens.
// Fitted to both scans of 8 to 61 sequences of 16 to 2048 tokens, in units of 16 tokens of 16 columns token by token (kCkUnitNs a key
// row: 1.9 us on the GPU for 16 heads of 128 x 128, delta rule): 0.77 a chunk and 1.03 a sequence here, 1 and 0.41 there, within 10 %.
// So the mean length should be 48, unless the chain of the longest sequence outlasts the work.  Us in chunks | by token, delta rule, 16
// heads, 60 sequences beside one: 32 tokens, 256: 330 | 305; 32, 1024: 398 | 389; 32, 2048: 490 | 526; 100, 256: 761 | 759; time mixing,
// 32 heads of 64: 123 | 118, 148 | 168, 201 | 296, 274 | 293.
constexpr int kCkMinTokens[2] = {256, 128};
constexpr int kCkMinMean = 48;
constexpr float kCkUnitNs[2] = {0.091f, 0.118f}, kCkTokenUs[2] = {0.13f, 0.26f};
constexpr long long kCkMaxBytes = 512ll << 20;
constexpr int kCkMinRound = 4;

struct ChunkPlan {
  bool fits;
  int dp, chunks, round;        // padded key rows; chunks of the longest sequence; chunks of a round
  bool by_tokens;
  int records;                  // of a head, counted by tokens
  long long rec_floats, carry_floats;
};

static int rec_floats(int mode, int dp) {
  if (mode == kDelta) return dp == 64 ? Rec<kDelta, 64>::kFloats : Rec<kDelta, 128>::kFloats;
  return dp == 64 ? Rec<kWkv, 64>::kFloats : Rec<kWkv, 128>::kFloats;
}

static ChunkPlan chunk_plan(int mode, int n, int n_seq, int max_len, int H, int d, int dv) {
  ChunkPlan p{};
  p.dp = d <= 64 ? 64 : 128;
  const float units = 0.77f * (n / kCk + n_seq / 2) + 1.03f * n_seq;
  const float work_us = units * H * ((dv + kCkCols - 1) / kCkCols) * kCkUnitNs[mode] * p.dp * 1e-3f;
  p.fits = max_len >= kCkMinTokens[mode] && d <= 128 && dv % 8 == 0 &&
           (n >= (long long)kCkMinMean * n_seq || max_len * kCkTokenUs[mode] > work_us);
  if (!p.fits) return p;
  p.chunks = (max_len + kCk - 1) / kCk;
  p.records = n / kCk + n_seq;
  const long long per = (long long)H * rec_floats(mode, p.dp), all = p.records * per;
  p.by_tokens = all * 4 <= kCkMaxBytes;
  if (p.by_tokens) {
    p.round = p.chunks;
    p.rec_floats = all;
  } else {
    p.carry_floats = (long long)n_seq * H * dv * p.dp;
    const long long r = (kCkMaxBytes / 4 - p.carry_floats) / (per * n_seq);
    p.fits = r >= kCkMinRound;
    p.round = (int)(r > p.chunks ? p.chunks : r);
    p.rec_floats = (long long)n_seq * p.round * per;
  }
  return p;
}

template <int MODE, typename T, int DP>
static int launch_chunks(ChunkArgs a, const ChunkPlan& p, int n_seq, cudaStream_t stream) {
  auto scan = chunk_scan_kernel<MODE, T, DP>;
  constexpr int bytes = ScanSmem<MODE, DP>::kBytes;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(scan, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  a.per_seq = p.by_tokens ? 0 : p.round;
  for (int c0 = 0; c0 < p.chunks; c0 += p.round) {
    a.c0 = c0;
    a.c1 = c0 + p.round;
    a.final = a.c1 >= p.chunks;
    const int now = p.chunks - c0 < p.round ? p.chunks - c0 : p.round;
    const dim3 records = p.by_tokens ? dim3(p.records, a.H) : dim3(now, a.H, n_seq);
    chunk_prepare_kernel<MODE, T, DP><<<records, DP, 0, stream>>>(a);
    scan<<<dim3((a.dv + kCkCols - 1) / kCkCols, a.H, n_seq), ScanSmem<MODE, DP>::kThreads, bytes, stream>>>(a);
  }
  return launch_status();
}

template <int MODE, typename T>
static int run_chunks(const ChunkArgs& a, const ChunkPlan& p, int n_seq, cudaStream_t stream) {
  if (p.dp == 64) return launch_chunks<MODE, T, 64>(a, p, n_seq, stream);
  return launch_chunks<MODE, T, 128>(a, p, n_seq, stream);
}

}  // namespace ell

using namespace ell;

// Floats of work space of a call in chunks, 0 where it goes token by token.  mode: 0 time mixing, 1 delta rule.
ELL_API long long ell_scan_chunks_work(int mode, int n, int n_seq, int max_len, int H, int d, int dv) {
  const ChunkPlan p = chunk_plan(mode, n, n_seq, max_len, H, d, dv);
  return p.fits ? p.rec_floats + p.carry_floats : 0;
}

// Arguments as those of ell_wkv_scan (mode 0; beta null) and ell_delta_scan (mode 1; u null, fp32, ldq = ldk = G d, ldv = H dv); n
// tokens in all; max_len sizes the launches: a longer sequence goes token by token from there on.  work: ell_scan_chunks_work floats on a 16-byte boundary.  v: rows of 16-byte pieces.
ELL_API int ell_scan_chunks(int mode, const void* q, const void* k, const void* v, const float* decay, const float* beta,
                            const float* u, float* o, float* state, const int* cu, const int* slots, const int* pos0, int n,
                            int n_seq, int max_len, int H, int G, int d, int dv, int ldq, int ldk, int ldv, int is_bf16, float* work,
                            int* err, cudaStream_t stream) {
  if (n_seq <= 0 || n <= 0) return 0;
  const ChunkPlan p = chunk_plan(mode, n, n_seq, max_len, H, d, dv);
  const int esz = is_bf16 ? 2 : 4;
  if (!p.fits || H % G || n_seq > 65535 || H > 65535 || (mode == kDelta && is_bf16)) return -2;
  if (work == nullptr || !aligned_to(work, 16) || !aligned_to(v, 16) || ldv * esz % 16 || dv * esz % 16) return -2;
  ChunkArgs a{q, k, v, decay, beta, u, o, state, cu, slots, pos0, work, p.carry_floats ? work + p.rec_floats : nullptr,
              H, G, d, dv, ldq, ldk, ldv, n_seq, 0, 0, 0, 1, err};
  if (mode == kDelta) return run_chunks<kDelta, float>(a, p, n_seq, stream);
  return is_bf16 ? run_chunks<kWkv, __nv_bfloat16>(a, p, n_seq, stream) : run_chunks<kWkv, float>(a, p, n_seq, stream);
}
