// Attention of single query rows over key/value rows: decoding from the cache, continued prompts, fp32 runs and head
// sizes the tcgen05 prefill kernel does not take.  GQA, value heads of their own size, ALiBi, a sink per head.
//
// Query row t sees the rows base[t] .. base[t] + len[t] - 1 of k [R, G, d] and v [R, G, dv] and sits at the last one.
// A CTA of 128 threads takes (row t, kv head, a range of keys) with all `rep` query heads of that kv head (in groups of
// at most 8), so every key and value is read once per group.  Tiles of KT keys and values come through two
// shared-memory stages (cp.async, the next tile in flight during the arithmetic).  Eight lanes share a key for the
// scores, the softmax runs on the KT scores of a head per warp, and for the weighted sum a thread owns eight value
// columns and a share of the tile's keys; the shares are added up once, at the end.  With more than one range per row a
// second kernel merges the partial (max, sum, accumulator) triples; the sink joins the denominator at the end, once.
// A window keeps the last `window` of a row's keys.  A gate multiplies head h's output of row t by sigmoid(gate[t][h]).
//
// Latent attention (one key row shared by all query heads, whose first dv columns are also the value, bf16) has a
// kernel of its own, attn_latent_kernel: the products run on mma.sync m16n8k16 over a key tile that is read once.
#include <algorithm>

#include "sm100.cuh"
#include "vec.cuh"

namespace ell {

constexpr int kArThreads = 128, kArRep = 8;   // kArRep: most query heads of a CTA (REP: 4 or 8)

struct AttnRowsArgs {
  const void *q, *k, *v;
  void* out;                      // [n, H, dv]
  float* part;                    // [n, H, splits, dv + 2] when splits > 1
  const int *base, *len;
  const float *sink, *slopes;
  int n, H, G, d, dv, ldq, ldk, ldv, splits, range;
  float scale;
  int window;                     // keys a row sees at most (INT_MAX: all)
  const void* gate;               // [n, ldg] of the activation type, or null
  int ldg;
  int* err;                       // error word (latent kernel)
  int all_ranges;                 // every range has a triple of every row
};

// Keys row t sees: the last min(len, window) of its rows.
struct RowKeys {
  size_t base;
  int len;
};
__device__ __forceinline__ RowKeys row_keys(const AttnRowsArgs& a, int t) {
  const int all = a.len[t], len = min(all, a.window);
  return {(size_t)a.base[t] + (all - len), len};
}
template <typename T>
__device__ __forceinline__ float row_gate(const AttnRowsArgs& a, int t, int h) {
  return a.gate == nullptr ? 1.f : sigmoid_f(to_f<T>(reinterpret_cast<const T*>(a.gate)[(size_t)t * a.ldg + h]));
}

// Shared memory: scaled queries [8][dp] | scores [8][KT] | statistics [8][4] | two stages of KT key rows, KT value rows.
struct ArLayout {
  int dp, krow, vrow, kgroups;    // padded key size; row strides in elements; key shares of the weighted sum
  int stage, bytes;               // elements of a stage; total bytes
};
__host__ __device__ inline ArLayout ar_layout(int d, int dv, int esz, int KT, int REP) {
  ArLayout l;
  l.dp = (d + 63) / 64 * 64;
  l.krow = l.dp + 16 / esz;
  const int oct = (dv + 7) / 8;
  l.vrow = oct * 8 + 16 / esz;
  l.kgroups = 1;
  while (2 * l.kgroups * oct <= kArThreads && 2 * l.kgroups <= KT / 4 && l.kgroups < 16) l.kgroups *= 2;
  l.stage = KT * (l.krow + l.vrow);
  const int head = (REP * l.dp + REP * KT + REP * 4) * 4;
  const int a = 2 * l.stage * esz, b = l.kgroups * REP * oct * 8 * 4;   // the sums reuse the stages
  l.bytes = head + (a > b ? a : b);
  return l;
}

template <typename T, int KT, int REP, bool VEC>
__global__ void __launch_bounds__(kArThreads) attn_rows_kernel(const AttnRowsArgs a) {
  chain_enter();
  extern __shared__ __align__(16) float sm[];
  const ArLayout L = ar_layout(a.d, a.dv, sizeof(T), KT, REP);
  const int t = blockIdx.x, rep = a.H / a.G, groups = (rep + REP - 1) / REP;
  const int g = blockIdx.y / groups, h0 = g * rep + (blockIdx.y % groups) * REP;
  const int nh = min(REP, g * rep + rep - h0);
  const int split = blockIdx.z, dp = L.dp, oct = (a.dv + 7) / 8;
  float* qs = sm;
  float* p = qs + REP * dp;
  float* stat = p + REP * KT;                    // max, sum, rescale
  T* stages = reinterpret_cast<T*>(stat + REP * 4);
  const RowKeys rk = row_keys(a, t);
  const int len = rk.len;
  const size_t base = rk.base;
  const int k0 = split * a.range, k1 = min(k0 + a.range, len);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // rows and columns the copies leave out must read as zero
  for (int i = threadIdx.x; i < 2 * L.stage * (int)sizeof(T) / 16; i += kArThreads)
    reinterpret_cast<uint4*>(stages)[i] = make_uint4(0, 0, 0, 0);
  for (int i = threadIdx.x; i < REP * dp; i += kArThreads) {
    const int h = i / dp, c = i % dp;
    qs[i] = h < nh && c < a.d
                ? to_f<T>(reinterpret_cast<const T*>(a.q)[(size_t)t * a.ldq + (size_t)(h0 + h) * a.d + c]) * a.scale : 0.f;
  }
  if (threadIdx.x < REP) {
    stat[threadIdx.x * 4] = -INFINITY;
    stat[threadIdx.x * 4 + 1] = 0.f;
  }
  __syncthreads();
  const T* kb = reinterpret_cast<const T*>(a.k) + base * a.ldk + (size_t)g * a.d;
  const T* vb = reinterpret_cast<const T*>(a.v) + base * a.ldv + (size_t)g * a.dv;
  auto load_tile = [&](int kt, int buf) {
    T* ks = stages + buf * L.stage;
    T* vs = ks + KT * L.krow;
    const int cnt = min(KT, k1 - kt);
    if (VEC) {
      constexpr int per = 16 / sizeof(T);
      const int kp = a.d / per, vp = a.dv / per;
      for (int i = threadIdx.x; i < cnt * kp; i += kArThreads) {
        const int r = i / kp, c = (i % kp) * per;
        cp_async16(ks + r * L.krow + c, kb + (size_t)(kt + r) * a.ldk + c);
      }
      for (int i = threadIdx.x; i < cnt * vp; i += kArThreads) {
        const int r = i / vp, c = (i % vp) * per;
        cp_async16(vs + r * L.vrow + c, vb + (size_t)(kt + r) * a.ldv + c);
      }
    } else {
      for (int i = threadIdx.x; i < cnt * a.d; i += kArThreads)
        ks[i / a.d * L.krow + i % a.d] = kb[(size_t)(kt + i / a.d) * a.ldk + i % a.d];
      for (int i = threadIdx.x; i < cnt * a.dv; i += kArThreads)
        vs[i / a.dv * L.vrow + i % a.dv] = vb[(size_t)(kt + i / a.dv) * a.ldv + i % a.dv];
    }
    cp_async_commit();
  };
  // weighted sum: this thread's eight columns and its share of a tile's keys
  const int my_oct = threadIdx.x % oct, my_share = threadIdx.x / oct, share = KT / L.kgroups;
  const bool adds = my_share < L.kgroups;
  float acc[REP][8];
#pragma unroll
  for (int h = 0; h < REP; ++h)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[h][j] = 0.f;
  const int l8 = lane & 7, grp = warp * 4 + (lane >> 3);          // 16 groups of 8 lanes
  constexpr int KJ = KT / 16;
  if (k0 < k1) load_tile(k0, 0);
  int buf = 0;
  for (int kt = k0; kt < k1; kt += KT, buf ^= 1) {
    if (kt + KT < k1) {
      load_tile(kt + KT, buf ^ 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const T* ks = stages + buf * L.stage;
    const T* vs = ks + KT * L.krow;
    // scores: a group takes keys grp, grp + 16, ...
    float sc[REP][KJ];
#pragma unroll
    for (int h = 0; h < REP; ++h)
#pragma unroll
      for (int j = 0; j < KJ; ++j) sc[h][j] = 0.f;
    for (int c = l8 * 8; c < dp; c += 64) {
      float kv[KJ][8];
#pragma unroll
      for (int j = 0; j < KJ; ++j) load_v<8>(ks + (grp + 16 * j) * L.krow + c, kv[j]);
#pragma unroll
      for (int h = 0; h < REP; ++h) {
        if (h < nh) {
          const float4 q0 = *reinterpret_cast<const float4*>(qs + h * dp + c);
          const float4 q1 = *reinterpret_cast<const float4*>(qs + h * dp + c + 4);
#pragma unroll
          for (int j = 0; j < KJ; ++j) {
            float s = sc[h][j];
            s = fmaf(q0.x, kv[j][0], s); s = fmaf(q0.y, kv[j][1], s); s = fmaf(q0.z, kv[j][2], s); s = fmaf(q0.w, kv[j][3], s);
            s = fmaf(q1.x, kv[j][4], s); s = fmaf(q1.y, kv[j][5], s); s = fmaf(q1.z, kv[j][6], s); s = fmaf(q1.w, kv[j][7], s);
            sc[h][j] = s;
          }
        }
      }
    }
#pragma unroll
    for (int h = 0; h < REP; ++h) {
      if (h < nh) {
#pragma unroll
        for (int j = 0; j < KJ; ++j) {
          float s = sc[h][j];
          s += __shfl_xor_sync(0xffffffffu, s, 1);
          s += __shfl_xor_sync(0xffffffffu, s, 2);
          s += __shfl_xor_sync(0xffffffffu, s, 4);
          const int key = kt + grp + 16 * j;
          if (l8 == 0) {
            if (a.slopes != nullptr) s += a.slopes[h0 + h] * (float)(key - (len - 1));
            p[h * KT + grp + 16 * j] = key < k1 ? s : -INFINITY;
          }
        }
      }
    }
    __syncthreads();
    for (int h = warp; h < nh; h += 4) {
      float s[(KT + 31) / 32], mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < (KT + 31) / 32; ++j) {
        s[j] = 32 * j + lane < KT ? p[h * KT + 32 * j + lane] : -INFINITY;
        mx = fmaxf(mx, s[j]);
      }
      const float m_old = stat[h * 4], m = fmaxf(m_old, warp_max(mx));   // finite: the tile has a key
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < (KT + 31) / 32; ++j) {
        const float e = expf(s[j] - m);
        sum += e;
        if (32 * j + lane < KT) p[h * KT + 32 * j + lane] = e;
      }
      sum = warp_sum(sum);
      if (lane == 0) {
        const float al = expf(m_old - m);
        stat[h * 4] = m;
        stat[h * 4 + 1] = stat[h * 4 + 1] * al + sum;
        stat[h * 4 + 2] = al;
      }
    }
    __syncthreads();
    if (adds) {
#pragma unroll
      for (int h = 0; h < REP; ++h) {
        if (h < nh) {
          const float al = stat[h * 4 + 2];
          if (al != 1.f) {
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[h][j] *= al;
          }
        }
      }
      const T* vp = vs + (size_t)(my_share * share) * L.vrow + my_oct * 8;
      for (int i = 0; i < share; i += 4) {
        float vv[4][8];
#pragma unroll
        for (int x = 0; x < 4; ++x) load_v<8>(vp + (i + x) * L.vrow, vv[x]);
#pragma unroll
        for (int h = 0; h < REP; ++h) {
          if (h < nh) {
            const float4 w = *reinterpret_cast<const float4*>(p + h * KT + my_share * share + i);
#pragma unroll
            for (int j = 0; j < 8; ++j)
              acc[h][j] = fmaf(w.w, vv[3][j], fmaf(w.z, vv[2][j], fmaf(w.y, vv[1][j], fmaf(w.x, vv[0][j], acc[h][j]))));
          }
        }
      }
    }
    __syncthreads();
  }
  // add the shares up: sums[share][head][column] over the stages' memory
  float* sums = reinterpret_cast<float*>(stages);
  if (adds) {
#pragma unroll
    for (int h = 0; h < REP; ++h)
      if (h < nh) store_v<8>(sums + ((my_share * REP + h) * oct + my_oct) * 8, acc[h]);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nh * a.dv; i += kArThreads) {
    const int h = i / a.dv, c = i % a.dv;
    float o = 0.f;
    for (int x = 0; x < L.kgroups; ++x) o += sums[(x * REP + h) * oct * 8 + c];
    const float m = stat[h * 4], l = stat[h * 4 + 1];
    if (a.splits == 1) {
      float den = l, f = 1.f;
      if (a.sink != nullptr) {
        const float sk = a.sink[h0 + h], mm = fmaxf(m, sk);
        f = expf(m - mm);
        den = l * f + expf(sk - mm);
      }
      reinterpret_cast<T*>(a.out)[((size_t)t * a.H + h0 + h) * a.dv + c] = from_f<T>(o * f / den * row_gate<T>(a, t, h0 + h));
    } else {
      float* pt = a.part + (((size_t)t * a.H + h0 + h) * a.splits + split) * (a.dv + 2);
      if (c == 0) {
        pt[0] = m;
        pt[1] = l;
      }
      pt[2 + c] = o;
    }
  }
}

// One CTA per (row, head): merge the ranges' triples.  Empty ranges carry max = -inf, sum = 0.  The ranges' weights are
// formed once (a range a thread), then every thread sums its columns over the ranges with independent loads.
constexpr int kArMaxSplits = 64;
template <typename T>
__global__ void __launch_bounds__(kArThreads) attn_rows_merge_kernel(const AttnRowsArgs a) {
  chain_enter();
  __shared__ float weight[kArMaxSplits];
  const int t = blockIdx.x, h = blockIdx.y, step = a.dv + 2;
  const float* pt = a.part + ((size_t)t * a.H + h) * a.splits * step;
  const int used = a.all_ranges ? a.splits : min(a.splits, (row_keys(a, t).len + a.range - 1) / a.range);
  if (threadIdx.x < 32) {
    const int s0 = threadIdx.x, s1 = threadIdx.x + 32;
    const float m0 = s0 < used ? pt[(size_t)s0 * step] : -INFINITY, m1 = s1 < used ? pt[(size_t)s1 * step] : -INFINITY;
    const float l0 = s0 < used ? pt[(size_t)s0 * step + 1] : 0.f, l1 = s1 < used ? pt[(size_t)s1 * step + 1] : 0.f;
    const float sk = a.sink != nullptr ? a.sink[h] : -INFINITY;
    const float m = fmaxf(warp_max(fmaxf(m0, m1)), sk);            // finite: the first range has a key
    const float e0 = expf(m0 - m), e1 = expf(m1 - m);
    const float den = warp_sum(l0 * e0 + l1 * e1) + (a.sink != nullptr ? expf(sk - m) : 0.f);
    const float f = row_gate<T>(a, t, h) / den;
    weight[s0] = e0 * f;
    weight[s1] = e1 * f;
  }
  __syncthreads();
  T* out = reinterpret_cast<T*>(a.out) + ((size_t)t * a.H + h) * a.dv;
  if (a.dv % 2 == 0) {                                             // triples start at even places
    for (int c = threadIdx.x * 2; c < a.dv; c += 2 * kArThreads) {
      float2 o = make_float2(0.f, 0.f);
#pragma unroll 8
      for (int s = 0; s < used; ++s) {
        const float2 v = *reinterpret_cast<const float2*>(pt + (size_t)s * step + 2 + c);
        o.x = fmaf(v.x, weight[s], o.x);
        o.y = fmaf(v.y, weight[s], o.y);
      }
      out[c] = from_f<T>(o.x);
      out[c + 1] = from_f<T>(o.y);
    }
  } else {
    for (int c = threadIdx.x; c < a.dv; c += kArThreads) {
      float o = 0.f;
#pragma unroll 8
      for (int s = 0; s < used; ++s) o = fmaf(pt[(size_t)s * step + 2 + c], weight[s], o);
      out[c] = from_f<T>(o);
    }
  }
}

// ---- latent attention: all heads share one key row, its first dv columns are the value ---------------
// A CTA of 16 warps takes (row t, 16 * MT query heads, a range of keys).  Tiles of 64 key rows come through two
// shared-memory stages as TMA boxes of 64 columns (128-byte swizzle: ldmatrix meets no bank conflicts).
//   scores   a warp multiplies 16 heads with 32 keys over one of 8 / MT slices of the columns (k-steps of 16); the
//            slices' sums go to shared memory in fp32
//   softmax  a warp owns MT heads, 32 / MT lanes each; fp32 weights, their sum unrounded, the operand of P·V in bf16
//   values   warp w owns columns [w, w + 1) * dv / 16 of all heads; the value operand is the key tile itself (ldmatrix
//            with transposition); its rescaled accumulators stay in registers
constexpr int kAlWarps = 16, kAlKeys = 64, kAlPStride = kAlKeys + 8, kAlSStride = kAlKeys + 4, kAlMaxNt = 4;
constexpr int kAlSRows = 8 * 16;                 // slices of the score product x heads
constexpr int kAlErr = 14;

constexpr int kAlBoxBytes = kAlKeys * 128;             // [64 keys x 64 columns]
__host__ __device__ inline int al_krow(int d) { return (d + 15) / 16 * 16 + 8; }       // stride of a query row
static int al_bytes(int d, int MT) {
  return 1024 + 2 * ((d + 63) / 64) * kAlBoxBytes + 16 * MT * (al_krow(d) * 2 + kAlPStride * 2 + 16) +
         kAlSRows * kAlSStride * 4 + 32;
}
// Place of a 16-byte piece (8 columns) of a key row in a stage.
__device__ __forceinline__ uint32_t al_place(int row, int piece) {
  return (uint32_t)((piece >> 3) * kAlBoxBytes + row * 128 + (((piece & 7) ^ (row & 7)) << 4));
}

__device__ __forceinline__ void ldsm4(uint32_t* r, const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void ldsm4_t(uint32_t* r, const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void mma_bf16(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// The same with a sum that starts here.
__device__ __forceinline__ void mma_bf16_first(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}

template <int MT>
__global__ void __launch_bounds__(kAlWarps * 32)
attn_latent_kernel(const __grid_constant__ CUtensorMap tmK, const AttnRowsArgs a) {
  chain_enter();
  extern __shared__ uint8_t alsm_raw[];
  uint8_t* kv = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(alsm_raw) + 1023) & ~(uintptr_t)1023);
  constexpr int HM = 16 * MT;
  const int krow = al_krow(a.d), dp = krow - 8, boxes = (a.d + 63) / 64, stage_bytes = boxes * kAlBoxBytes;
  __nv_bfloat16* qs = reinterpret_cast<__nv_bfloat16*>(kv + 2 * stage_bytes);
  __nv_bfloat16* ps = qs + HM * krow;
  float* ss = reinterpret_cast<float*>(ps + HM * kAlPStride);
  float* stat = ss + kAlSRows * kAlSStride;                  // max | sum | rescale, HM each
  uint64_t* full = reinterpret_cast<uint64_t*>(stat + 4 * HM);      // one barrier a stage
  int* gave_up = reinterpret_cast<int*>(full + 2);
  const int t = blockIdx.x, h0 = blockIdx.y * HM, nh = min(HM, a.H - h0), split = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const RowKeys rk = row_keys(a, t);
  const int k0 = split * a.range, k1 = min(k0 + a.range, rk.len);
  const __nv_bfloat16* qb = reinterpret_cast<const __nv_bfloat16*>(a.q) + (size_t)t * a.ldq + (size_t)h0 * a.d;
  const int pieces = a.d / 8, padded = dp / 8;         // 16-byte pieces of a row
  const int tail = k1 > k0 ? (k1 - k0 - 1) % kAlKeys + 1 : kAlKeys, tiles = k1 > k0 ? (k1 - k0 + kAlKeys - 1) / kAlKeys : 0;
  // one thread: columns past d and rows past the tensor are zero-filled
  auto load_tile = [&](int kt, int buf) {
    sm100::mbar_expect_tx(&full[buf], (uint32_t)stage_bytes);
    for (int c = 0; c < boxes; ++c)
      sm100::tma_load_2d(kv + buf * stage_bytes + c * kAlBoxBytes, &tmK, &full[buf], c * 64, (int)rk.base + kt);
  };
  if (threadIdx.x == 0) {
    sm100::mbar_init(&full[0], 1);
    sm100::mbar_init(&full[1], 1);
    *gave_up = *(volatile int*)a.err;                  // an earlier kernel already failed: do not wait on anything
    sm100::fence_barrier_init();
    if (tiles > 0 && *gave_up == 0) load_tile(k0, 0);  // on its way while the queries come
  }
  // query rows and columns past the end read as zero
  for (int i = threadIdx.x; i < HM * padded; i += kAlWarps * 32) {
    const int h = i / padded, c = i % padded;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (h < nh && c < pieces) v = *reinterpret_cast<const uint4*>(qb + (size_t)h * a.d + c * 8);
    *reinterpret_cast<uint4*>(qs + h * krow + c * 8) = v;
  }
  if (threadIdx.x < HM) {
    stat[threadIdx.x] = -INFINITY;
    stat[HM + threadIdx.x] = 0.f;
    stat[2 * HM + threadIdx.x] = 1.f;
  }
  const int nt = (a.dv / 8 + kAlWarps - 1) / kAlWarps;         // 8-column pieces of a warp
  const int col0 = warp * nt * 8, mine = max(0, min(nt, (a.dv - col0) / 8));
  float acc[MT][kAlMaxNt][4];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int n = 0; n < kAlMaxNt; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[m][n][i] = 0.f;
  const int g = lane >> 2, tq = lane & 3;
  const int l8 = lane & 7, quad = lane >> 3;
  __syncthreads();
  const bool dead = *gave_up != 0;
  constexpr int KS = 8 / MT;                             // column slices of the score product
  const int mt = MT == 1 ? 0 : warp >> 3, key0 = (warp & 1) * 32, slice = (warp >> 1) % KS;
  for (int it = 0; it < tiles && !dead; ++it) {
    const int buf = it & 1, kt = k0 + it * kAlKeys;
    uint8_t* ks = kv + buf * stage_bytes;
    if (threadIdx.x == 0 && it + 1 < tiles) load_tile(kt + kAlKeys, buf ^ 1);   // the end of the last step freed that stage
    if (!sm100::mbar_wait(&full[buf], (it >> 1) & 1, gave_up)) *(volatile int*)gave_up = 1;
    else if (it == tiles - 1)                            // rows past the range are other keys: their weight is 0, not their value
      for (int i = threadIdx.x; i < (kAlKeys - tail) * padded; i += kAlWarps * 32)
        *reinterpret_cast<uint4*>(ks + al_place(tail + i / padded, i % padded)) = make_uint4(0, 0, 0, 0);
    __syncthreads();
    if (*(volatile int*)gave_up) {
      if (threadIdx.x == 0) {
        atomicCAS(a.err, 0, kAlErr);
        const unsigned long long t0 = sm100::globaltimer_ns();          // copies still in flight land before the CTA ends
        while (sm100::globaltimer_ns() - t0 < 200000ull) {
        }
      }
      __syncthreads();
      break;                                             // uniform: every thread reads the flag after the barrier
    }
    // scores of 16 heads and 32 keys over this warp's slice of the columns
    {
      float sc[4][4];
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) sc[n][i] = 0.f;
      const __nv_bfloat16* qrow = qs + (mt * 16 + (quad & 1) * 8 + l8) * krow + (quad >> 1) * 8;
      const int krow_i = key0 + (quad >> 1) * 8 + l8;
#pragma unroll 3
      for (int c = slice * 16; c < dp; c += KS * 16) {
        uint32_t a0[4], b0[4], b1[4];
        ldsm4(a0, qrow + c);
        const uint32_t at = al_place(krow_i, (c >> 3) + (quad & 1));       // 16 rows on: the same swizzle
        ldsm4(b0, ks + at);
        ldsm4(b1, ks + at + 16 * 128);
        mma_bf16(sc[0], a0, b0[0], b0[1]);
        mma_bf16(sc[1], a0, b0[2], b0[3]);
        mma_bf16(sc[2], a0, b1[0], b1[1]);
        mma_bf16(sc[3], a0, b1[2], b1[3]);
      }
      float* dst = ss + (slice * HM + mt * 16 + g) * kAlSStride + key0 + tq * 2;
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        *reinterpret_cast<float2*>(dst + n * 8) = make_float2(sc[n][0], sc[n][1]);
        *reinterpret_cast<float2*>(dst + 8 * kAlSStride + n * 8) = make_float2(sc[n][2], sc[n][3]);
      }
    }
    __syncthreads();
    {
      constexpr int LH = 32 / MT, KL = kAlKeys / LH;       // lanes a head, keys a lane
      const int hh = warp * MT + lane / LH, key = (lane % LH) * KL;
      float sv[KL], mx = -INFINITY, sum = 0.f;
#pragma unroll
      for (int j = 0; j < KL; ++j) sv[j] = 0.f;
#pragma unroll
      for (int y = 0; y < KS; ++y) {
        const float* row = ss + (y * HM + hh) * kAlSStride + key;
#pragma unroll
        for (int j = 0; j < KL; j += 2) {
          const float2 v = *reinterpret_cast<const float2*>(row + j);
          sv[j] += v.x;
          sv[j + 1] += v.y;
        }
      }
#pragma unroll
      for (int j = 0; j < KL; ++j) {
        sv[j] = kt + key + j < k1 ? sv[j] * a.scale : -INFINITY;
        mx = fmaxf(mx, sv[j]);
      }
#pragma unroll
      for (int o = LH / 2; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      const float m_old = stat[hh], m = fmaxf(m_old, mx);  // finite: the tile has a key
#pragma unroll
      for (int j = 0; j < KL; ++j) {
        sv[j] = expf(sv[j] - m);
        sum += sv[j];
      }
#pragma unroll
      for (int j = 0; j < KL; j += 2)
        *reinterpret_cast<__nv_bfloat162*>(ps + hh * kAlPStride + key + j) = __floats2bfloat162_rn(sv[j], sv[j + 1]);
#pragma unroll
      for (int o = LH / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (lane % LH == 0) {                                // its lanes have read the old maximum: the shuffles above
        const float al = expf(m_old - m);
        stat[hh] = m;
        stat[HM + hh] = stat[HM + hh] * al + sum;
        stat[2 * HM + hh] = al;
      }
    }
    __syncthreads();
    uint32_t pa[MT][kAlKeys / 16][4];
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      const float r0 = stat[2 * HM + m * 16 + g], r1 = stat[2 * HM + m * 16 + g + 8];
#pragma unroll
      for (int n = 0; n < kAlMaxNt; ++n) {
        acc[m][n][0] *= r0;
        acc[m][n][1] *= r0;
        acc[m][n][2] *= r1;
        acc[m][n][3] *= r1;
      }
#pragma unroll
      for (int k = 0; k < kAlKeys / 16; ++k)
        ldsm4(pa[m][k], ps + (m * 16 + (quad & 1) * 8 + l8) * kAlPStride + k * 16 + (quad >> 1) * 8);
    }
#pragma unroll
    for (int n = 0; n < kAlMaxNt; ++n) {
      if (n < mine) {
#pragma unroll
        for (int k = 0; k < kAlKeys / 32; ++k) {         // 32 keys x 8 columns per ldmatrix
          uint32_t b[4];
          ldsm4_t(b, ks + al_place(k * 32 + quad * 8 + l8, col0 / 8 + n));
#pragma unroll
          for (int m = 0; m < MT; ++m) {
            mma_bf16(acc[m][n], pa[m][2 * k], b[0], b[1]);
            mma_bf16(acc[m][n], pa[m][2 * k + 1], b[2], b[3]);
          }
        }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int hh = m * 16 + g + r * 8;
      if (hh >= nh) continue;
      const size_t th = (size_t)t * a.H + h0 + hh;
      const float l = stat[HM + hh];
      if (a.splits == 1) {
        const float f = row_gate<__nv_bfloat16>(a, t, h0 + hh) / l;
        __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(a.out) + th * a.dv + col0 + tq * 2;
#pragma unroll
        for (int n = 0; n < kAlMaxNt; ++n)
          if (n < mine)
            *reinterpret_cast<__nv_bfloat162*>(o + n * 8) = __floats2bfloat162_rn(acc[m][n][2 * r] * f, acc[m][n][2 * r + 1] * f);
      } else {
        float* pt = a.part + (th * a.splits + split) * (a.dv + 2);
        if (warp == 0 && tq == 0) {
          pt[0] = stat[hh];
          pt[1] = l;
        }
#pragma unroll
        for (int n = 0; n < kAlMaxNt; ++n)
          if (n < mine) *reinterpret_cast<float2*>(pt + 2 + col0 + n * 8 + tq * 2) = make_float2(acc[m][n][2 * r], acc[m][n][2 * r + 1]);
      }
    }
}

// ---- bf16 rows over cached keys on matrix instructions ------------------------------------------------------------
// Decoding reads every cached key and value once for a few query rows: bound by those bytes, if the arithmetic keeps up.
// On the FMA pipe it did not (230 us for 64 rows x 2048 keys x 8 key heads, 537 MB, which take 83); and a continued prompt
// read its whole context once per token (1060 us for 301 tokens of two sequences over 3000).  Here a tile of rows is the consecutive
// tokens of one sequence times the query heads of one key head, and matrix instructions do the products:
//   scores  exact bf16 products, fp32 sums, scale and bias applied in fp32
//   values  the fp32 weights go in as three bf16 parts, so they keep their 24 bits.  The products of a few keys start from zero, the small
//           parts first, and are added to the sums in fp32: the tensor core cuts off what does not fit its accumulator, and a sum that
//           stays in one drifts with its length
//   attn_few_kernel   up to 16 rows (decoding), on mma.sync.  Keys are the M side of both products and rows the N side, so 8 rows
//                     cost half of 16: S^T = K q^T, O^T = V^T P^T.  The four warps take units of 16 keys in turn, each with a softmax,
//                     sums and a ring of three stages of its own, filled by TMA; no barrier until their results meet.
//                     Bound by the keys' and values' bytes.  us, merge included, one B200, keys larger than L2 (8 sequences: as large):
//                     64 rows x 2100 keys x 8 key heads, 551 MB, 87 (6.3 TB/s); 8 x 4200 x 8 29.4; 10 x 2048 x 32 62; one x 4000 x 4 9.7.
//                     With 16 cp.async and their addresses a lane and unit 117, 43, 82 and 10.6.  With ex2 of a rounded x log2(e) in
//                     place of expf and sums that stay in the accumulators 86, 28.8, 60 and 9.5, but 1.1e-6 off 64 bits in front of the
//                     rounding to bf16, and 3.3e-6 for values of one sign, where this is 2.1e-7 and 5e-8 (8 x 4200).  Equal shares of
//                     all keys for every CTA, rows divided where a share ends: 92, 31 and 14 (the last for one x 4000).
//   attn_tile_kernel  more rows (continued prompts): 128 of them on tcgen05, see there
// Ranges of keys and their merge are those of attn_rows_kernel.
constexpr int kAtThreads = 128;
constexpr int kAtHeads = 16;                                       // most query heads of a CTA
constexpr int kAfKeys = 16, kAfChunk = kAfKeys * 128;              // keys of a warp's unit; bytes of 64 columns of them
// All of a CTA's shared memory is in kAfSmem: two CTAs and the system's 1 KB each just fit a split of 196 KB.  112 bytes more took 228 KB,
// which later kernels of the chain found their L1 cut down by (a decoding product of 6144 x 4096 13.6 -> 19.5 us).
constexpr int kAfStage = 4 * kAfChunk, kAfStages = 3, kAfRing = 4 * kAfStages * kAfStage, kAfSmem = kAfRing + 1024;
static_assert(2 * (kAfSmem + 1024) <= 196 * 1024, "");
constexpr int kAfErr = 18;

// x and y as three bf16 parts each, eight of their 24 bits a part: nothing is lost.  By truncation, since conversions share the unit of
// the exponential.
__device__ __forceinline__ void cut_bf16(float x, float y, uint32_t (&p)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    p[i] = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
    x -= __uint_as_float(__float_as_uint(x) & 0xffff0000u);
    y -= __uint_as_float(__float_as_uint(y) & 0xffff0000u);
  }
}

// The tokens, heads and keys of a CTA.  blockIdx.x: tile of `tt` tokens of a sequence (cu null: one token each), y: key head
// and group of its query heads, z: range of keys.
struct AtTile {
  int r0, r1, g, h0, nh, rows, k0, k1, len0, last_first;
  size_t base;
  __device__ __forceinline__ bool init(const AttnRowsArgs& a, const int* cu, int tiles, int tt) {
    if (cu != nullptr) {
      const int seq = blockIdx.x / tiles;
      r0 = cu[seq] + blockIdx.x % tiles * tt;
      r1 = min(r0 + tt, cu[seq + 1]);
      if (r0 >= r1) return false;
    } else {
      r0 = blockIdx.x;
      r1 = r0 + 1;
    }
    const int rep = a.H / a.G, groups = (rep + kAtHeads - 1) / kAtHeads;
    g = blockIdx.y / groups;
    h0 = g * rep + blockIdx.y % groups * kAtHeads;
    nh = min(kAtHeads, (g + 1) * rep - h0);
    rows = (r1 - r0) * nh;
    base = a.base[r0];
    len0 = a.len[r0];
    const int len1 = a.len[r1 - 1];
    last_first = max(0, len1 - a.window);
    k0 = max(0, len0 - a.window) + (int)blockIdx.z * a.range;
    k1 = min(k0 + a.range, len1);
    return true;
  }
  __device__ __forceinline__ int token(int m) const { return r0 + m / nh; }
  __device__ __forceinline__ int head(int m) const { return h0 + m % nh; }
  // where row m goes: its place in `out` (with the factor of its sums), or the triple of this range
  __device__ __forceinline__ __nv_bfloat16* place(const AttnRowsArgs& a, int m, float mx, float l, float& f, float*& part) const {
    const size_t th = (size_t)token(m) * a.H + head(m);
    part = nullptr;
    f = 1.f;
    if (a.splits > 1) {
      part = a.part + (th * a.splits + blockIdx.z) * (a.dv + 2);
      return nullptr;
    }
    float den = l;
    if (a.sink != nullptr) {
      const float sk = a.sink[head(m)], mm = fmaxf(mx, sk);
      f = expf(mx - mm);
      den = l * f + expf(sk - mm);
    }
    f = f / den * row_gate<__nv_bfloat16>(a, token(m), head(m));
    return reinterpret_cast<__nv_bfloat16*>(a.out) + th * a.dv;
  }
};

__device__ __forceinline__ bool not_finite(float x) { return !(x * 0.f == 0.f); }

// Row m of the tile key by key, by one warp, with the keys that the row sees and no others.  In the tiles a key that a row does not
// see has the weight 0, and 0 times an infinity or NaN of a later token (or of one that left the window) is NaN; the bf16 parts of a
// weight times an infinity are of either sign.  A row that came out not finite is therefore computed again here (1 us a few keys).
__device__ __noinline__ void at_row_alone(const AttnRowsArgs& a, const AtTile T, int m) {
  const int lane = threadIdx.x & 31, tok = T.token(m), head = T.head(m), end = a.len[tok];
  const __nv_bfloat16* q = reinterpret_cast<const __nv_bfloat16*>(a.q) + (size_t)tok * a.ldq + (size_t)head * a.d;
  const float slope = a.slopes != nullptr ? a.slopes[head] : 0.f;
  float qv[4], acc[4], mx = -INFINITY, l = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    qv[i] = lane + 32 * i < a.d ? __bfloat162float(q[lane + 32 * i]) : 0.f;
    acc[i] = 0.f;
  }
  for (int key = max(T.k0, end - a.window); key < min(T.k1, end); ++key) {
    const __nv_bfloat16* k = reinterpret_cast<const __nv_bfloat16*>(a.k) + (T.base + key) * a.ldk + (size_t)T.g * a.d;
    const __nv_bfloat16* v = reinterpret_cast<const __nv_bfloat16*>(a.v) + (T.base + key) * a.ldv + (size_t)T.g * a.dv;
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (lane + 32 * i < a.d) s = fmaf(qv[i], __bfloat162float(k[lane + 32 * i]), s);
    s = warp_sum(s) * a.scale;
    if (a.slopes != nullptr) s += slope * (float)(key - (end - 1));
    const float now = fmaxf(mx, s), al = mx == now ? 1.f : expf(mx - now), w = s == -INFINITY ? 0.f : expf(s - now);
    mx = now;
    l = l * al + w;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (lane + 32 * i < a.dv) acc[i] = fmaf(w, __bfloat162float(v[lane + 32 * i]), acc[i] * al);
  }
  float f, *part;
  __nv_bfloat16* out = T.place(a, m, mx, l, f, part);
  if (part != nullptr && lane == 0) {
    part[0] = mx;
    part[1] = l;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (lane + 32 * i < a.dv) {
      if (part != nullptr) part[2 + lane + 32 * i] = acc[i];
      else out[lane + 32 * i] = __float2bfloat16_rn(acc[i] * f);
    }
}

__device__ __forceinline__ uint32_t transpose_8x8(uint32_t x) {
  uint32_t y;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
  return y;
}

struct AfRing {
  uint64_t full[4][kAfStages];    // of a warp's stages
  int gave_up;
};
static_assert(sizeof(AfRing) <= 128, "");
// The stages start at a multiple of 1024; the barriers lie in what is left in front of them, or behind.
__device__ __forceinline__ uint8_t* af_stages(uint8_t* raw) {
  return reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~(uintptr_t)1023);
}
__device__ __forceinline__ AfRing& af_ring(uint8_t* raw) {
  uint8_t* stages = af_stages(raw);
  return *reinterpret_cast<AfRing*>(stages - raw >= 128 ? raw : stages + kAfRing);
}
// NB: groups of 8 rows.  FULL: heads of 128.
template <int NB, bool FULL>
__global__ void __launch_bounds__(kAtThreads, 2)
attn_few_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const __grid_constant__ AttnRowsArgs a,
                const int* __restrict__ cu, int tiles, int tt) {
  extern __shared__ __align__(128) uint8_t atsm_raw[];
  uint8_t* atsm = af_stages(atsm_raw);
  AfRing& ring = af_ring(atsm_raw);
  if (threadIdx.x == 0) {
    for (int w = 0; w < 4; ++w)
      for (int i = 0; i < kAfStages; ++i) sm100::mbar_init(&ring.full[w][i], 1);
    sm100::fence_barrier_init();
    sm100::tma_prefetch_desc(&tmK);
    sm100::tma_prefetch_desc(&tmV);
    ring.gave_up = 0;
  }
  __syncthreads();
  chain_enter(cu);
  AtTile T;
  if (!T.init(a, cu, tiles, tt)) return;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31, gr = lane >> 2, t = lane & 3, quad = lane >> 3,
            l8 = lane & 7;
  uint8_t* stages = atsm + warp * kAfStage * kAfStages;
  const int n_units = T.k1 > T.k0 ? (T.k1 - T.k0 + kAfKeys - 1) / kAfKeys : 0;
  const int mine = n_units > warp ? (n_units - warp + 3) / 4 : 0;       // units warp, warp + 4, ...
  const int kc = FULL ? 2 : (a.d + 63) / 64, vc = FULL ? 2 : (a.dv + 63) / 64;
  volatile int* gave_up = &ring.gave_up;
  // rows past the range are whatever lies there: their weight is 0, and their values are cleared
  auto load = [&](int i) {
    if (i < mine && lane == 0) {
      const int s = i % kAfStages;
      uint8_t* st = stages + s * kAfStage;
      const int row = (int)T.base + T.k0 + (warp + 4 * i) * kAfKeys;
      sm100::mbar_expect_tx(&ring.full[warp][s], (kc + vc) * kAfChunk);
      for (int c = 0; c < kc; ++c) sm100::tma_load_3d(st + c * kAfChunk, &tmK, &ring.full[warp][s], c * 64, T.g, row);
      for (int c = 0; c < vc; ++c) sm100::tma_load_3d(st + (2 + c) * kAfChunk, &tmV, &ring.full[warp][s], c * 64, T.g, row);
    }
  };
#pragma unroll
  for (int i = 0; i < kAfStages - 1; ++i) load(i);

  const int ksteps = FULL ? 8 : a.d / 16, vtiles = FULL ? 8 : a.dv / 16;
  uint32_t q[NB][8][2];                              // B operand: row gr of the group
  float m[NB][2], l[NB][2], slope[NB][2];            // of rows 2 t, 2 t + 1: maximum, this lane's share of the sum
  int first[NB][2], end[NB][2];                      // keys they see
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    const int r = min(b * 8 + gr, T.rows - 1);       // rows past the end repeat the last
    const __nv_bfloat16* src = reinterpret_cast<const __nv_bfloat16*>(a.q) + (size_t)T.token(r) * a.ldq + (size_t)T.head(r) * a.d + 2 * t;
#pragma unroll
    for (int k = 0; k < 8; ++k)
#pragma unroll
      for (int c = 0; c < 2; ++c) q[b][k][c] = k < ksteps ? *reinterpret_cast<const uint32_t*>(src + k * 16 + c * 8) : 0u;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int n = min(b * 8 + 2 * t + j, T.rows - 1);
      end[b][j] = a.len[T.token(n)];
      first[b][j] = max(0, end[b][j] - a.window);
      slope[b][j] = a.slopes != nullptr ? a.slopes[T.head(n)] : 0.f;
      m[b][j] = -INFINITY;
      l[b][j] = 0.f;
    }
  }
  float acc[8][NB][4];                               // 16 value columns x 8 rows each
#pragma unroll
  for (int n = 0; n < 8; ++n)
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[n][b][i] = 0.f;

  constexpr int kTogether = 4 / NB;
  const uint32_t k_row = ((quad & 1) * 8 + l8) * 128, v_row = ((quad >> 1) * 8 + l8) * 128 + 2 * kAfChunk;      // row & 7 = l8
  bool failed = false;
  for (int i = 0; i < mine; ++i) {
    const int stage = i % kAfStages;
    failed = !sm100::mbar_wait_warp(&ring.full[warp][stage], (i / kAfStages) & 1, gave_up);
    if (failed) break;
    load(i + kAfStages - 1);                           // over the unit before, which all lanes are done with (the fence and the votes)
    const uint8_t *ks = stages + stage * kAfStage + k_row, *vs = stages + stage * kAfStage + v_row;
    const int key0 = T.k0 + (warp + 4 * i) * kAfKeys;
    if (key0 + kAfKeys > T.k1) {                       // 0 times what a former sequence left behind the end must be 0
      uint8_t* left = stages + stage * kAfStage + 2 * kAfChunk + (T.k1 - key0) * 128;
      const int pieces = (key0 + kAfKeys - T.k1) * 8;
      for (int c = 0; c < vc; ++c)
        for (int p = lane; p < pieces; p += 32) *reinterpret_cast<uint4*>(left + c * kAfChunk + p * 16) = make_uint4(0, 0, 0, 0);
      __syncwarp();
    }
    float s[NB][4], s2[NB][4];                       // two chains of sums
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
      for (int i = 0; i < 4; ++i) s[b][i] = s2[b][i] = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (k < ksteps) {
        uint32_t x[4];
        ldsm4(x, ks + (k >> 2) * kAfChunk + ((((k & 3) * 2 + (quad >> 1)) ^ l8) << 4));
#pragma unroll
        for (int b = 0; b < NB; ++b) mma_bf16(k & 1 ? s2[b] : s[b], x, q[b][k][0], q[b][k][1]);
      }
    }
    const bool mask = key0 + kAfKeys > min(T.len0, T.k1) || key0 < T.last_first;
    float al[NB][2];
#pragma unroll
    for (int b = 0; b < NB; ++b) {
#pragma unroll
      for (int i = 0; i < 4; ++i) s[b][i] = (s[b][i] + s2[b][i]) * a.scale;
      if (a.slopes != nullptr || mask) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int j = i & 1, key = key0 + gr + (i >> 1) * 8;
          s[b][i] += slope[b][j] * (float)(key - (end[b][j] - 1));
          if (key < first[b][j] || key >= end[b][j]) s[b][i] = -INFINITY;
        }
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        float mx = fmaxf(s[b][j], s[b][j + 2]);
#pragma unroll
        for (int o = 4; o <= 16; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float now = fmaxf(m[b][j], mx);
        al[b][j] = now == -INFINITY ? 1.f : expf(m[b][j] - now);       // no key yet: nothing to rescale
        m[b][j] = now;
        const float ref = now == -INFINITY ? 0.f : now;
        s[b][j] = expf(s[b][j] - ref);
        s[b][j + 2] = expf(s[b][j + 2] - ref);
        l[b][j] = l[b][j] * al[b][j] + (s[b][j] + s[b][j + 2]);
      }
    }
    uint32_t w[NB][2][3];                            // weights as the B operand: keys 2 t .. of row gr
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        cut_bf16(s[b][2 * c], s[b][2 * c + 1], w[b][c]);
#pragma unroll
        for (int x = 0; x < 3; ++x) w[b][c][x] = transpose_8x8(w[b][c][x]);
      }
#pragma unroll
    for (int n = 0; n < 8; n += kTogether) {
      // the parts' products of one accumulator wait for one another, so several accumulators take turns
      uint32_t x[kTogether][4];
#pragma unroll
      for (int y = 0; y < kTogether; ++y)
        if (n + y < vtiles) ldsm4_t(x[y], vs + ((n + y) >> 2) * kAfChunk + (((((n + y) & 3) * 2 + (quad & 1)) ^ l8) << 4));
      float sum[kTogether][NB][4];
#pragma unroll
      for (int i = 2; i >= 0; --i)
#pragma unroll
        for (int y = 0; y < kTogether; ++y)
          if (n + y < vtiles) {
#pragma unroll
            for (int b = 0; b < NB; ++b) {
              if (i == 2) mma_bf16_first(sum[y][b], x[y], w[b][0][i], w[b][1][i]);
              else mma_bf16(sum[y][b], x[y], w[b][0][i], w[b][1][i]);
            }
          }
#pragma unroll
      for (int y = 0; y < kTogether; ++y)
        if (n + y < vtiles) {
#pragma unroll
          for (int b = 0; b < NB; ++b)
#pragma unroll
            for (int i = 0; i < 4; i += 2) {
              float* o = acc[n + y][b] + i;
              const float2 v = sm100::ffma2(make_float2(o[0], o[1]), make_float2(al[b][0], al[b][1]), make_float2(sum[y][b][i], sum[y][b][i + 1]));
              o[0] = v.x;
              o[1] = v.y;
            }
        }
    }
    sm100::fence_proxy_async_smem();                   // these reads before the copies that go over them
    __syncwarp();
  }
#pragma unroll
  for (int b = 0; b < NB; ++b)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int o = 4; o <= 16; o <<= 1) l[b][j] += __shfl_xor_sync(0xffffffffu, l[b][j], o);

  if (failed) *gave_up = 1;
  __syncthreads();
  if (*gave_up) {                                      // copies in flight land before the CTA ends
    if (threadIdx.x == 0) {
      atomicCAS(a.err, 0, kAfErr);
      const unsigned long long t0 = sm100::globaltimer_ns();
      while (sm100::globaltimer_ns() - t0 < 200000ull) {
      }
    }
    __syncthreads();
    return;
  }
  float* stat = reinterpret_cast<float*>(atsm);      // [warp][16 rows] maximum | sum
  float* sums = stat + 128;                          // [warp][16 rows][ld]
  const int ld = a.dv + 8;
  if (gr == 0) {
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        stat[warp * 16 + b * 8 + 2 * t + j] = m[b][j];
        stat[64 + warp * 16 + b * 8 + 2 * t + j] = l[b][j];
      }
  }
#pragma unroll
  for (int n = 0; n < 8; ++n) {
    if (n < vtiles) {
#pragma unroll
      for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          sums[(size_t)(warp * 16 + b * 8 + 2 * t + (i & 1)) * ld + n * 16 + gr + (i >> 1) * 8] = acc[n][b][i];
    }
  }
  __syncthreads();
  for (int r = warp; r < T.rows; r += 4) {
    float mx = -INFINITY, sum = 0.f, w[4], f;
#pragma unroll
    for (int x = 0; x < 4; ++x) mx = fmaxf(mx, stat[x * 16 + r]);
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const float mw = stat[x * 16 + r];
      w[x] = mw == -INFINITY ? 0.f : expf(mw - mx);
      sum += w[x] * stat[64 + x * 16 + r];
    }
    float* part;
    __nv_bfloat16* out = T.place(a, r, mx, sum, f, part);
    if (part != nullptr && lane == 0) {
      part[0] = mx;
      part[1] = sum;
    }
    bool odd = not_finite(sum);
    for (int c = lane * 2; c < a.dv; c += 64) {
      float2 o = make_float2(0.f, 0.f);
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const float2 v = *reinterpret_cast<const float2*>(sums + (size_t)(x * 16 + r) * ld + c);
        o.x = fmaf(w[x], v.x, o.x);
        o.y = fmaf(w[x], v.y, o.y);
      }
      odd |= not_finite(o.x) || not_finite(o.y);
      if (part != nullptr) *reinterpret_cast<float2*>(part + 2 + c) = o;
      else *reinterpret_cast<__nv_bfloat162*>(out + c) = __floats2bfloat162_rn(o.x * f, o.y * f);
    }
    odd = __any_sync(0xffffffffu, odd);
    __syncwarp();
    if (odd) at_row_alone(a, T, r);
  }
}

// ---- continued prompts on tcgen05 ----------------------------------------------------------------------
// A CTA takes 128 rows (consecutive tokens of one sequence times the query heads of one key head) and a range of keys, in tiles of 64:
//   warps 0-7   softmax: a thread owns a row, its TMEM lane, and half of a tile's keys (warps 4-7 the second half; the maxima meet in
//               shared memory).  Fp32 weights go back to TMEM as three bf16 parts, so that the product with V keeps their 24 bits
//   warps 8-15  sums: a thread owns a row and half of its value columns in registers, and adds every tile's product to them in fp32
//   warp 16     issues: S = Q K^T (128 x 64), O_tile = P_2 V + P_1 V + P_0 V (P from TMEM, V in place as an MN-major operand)
//   warp 17     TMA: tiles of keys and values through a ring of four stages
// TMEM columns: for even and odd tiles S 0-63, P_0 and P_1 over the scores that the threads have read, P_2 64-95 (128-223); O_tile
// 256-383 and 384-511.
// Every tile's product starts from zero, the small parts first, so that four products of it are cut at the tile's own size, and no
// accumulator is read back to be rescaled.  512 tokens over 4096 keys, in fp32 in front of the rounding to bf16, against 64 bits: 3.2e-7, and
// 1.1e-7 for values of one sign; with sums that stay in TMEM and ex2 of a rounded x log2(e) 7.3e-6 and 2.3e-5, with mma.sync's
// accumulators 4.6e-6 and 4.8e-6.
// One CTA an SM; bound by the softmax, 1.5 us a tile (its twenty products take 0.55).  us, kernel and merge, one B200: 301 tokens of two
// sequences over 3000, 16 heads on 8, 41; 512 tokens over 4096, 32 on 8, 99; 512 over 1000 beside three of 16 tokens, 16 on 4, 33; 700 over
// 2000, 16 on 16, 54; 17 over 3000, 32 on 8, 18; 33 over 64 10.4; 64 over 1200, 16 heads of 64, 17.6.  Two CTAs an SM with 256 columns and 97 KB
// each, whose sums stayed in TMEM: 40, 106, 45, 54, 19, 9.5 and 15.3; a warp for 16 rows on mma.sync: 134, 466, 74, 150, 39, 10.8 and 20.8.
constexpr int kAtTile = 64, kAtRows = 128, kAtTileThreads = 576, kAtHalf = kAtTile / 2, kAtStages = 4;
constexpr int kAtQChunk = kAtRows * 128, kAtKvChunk = kAtTile * 128;     // [rows x 64 columns], 128-byte swizzle rows
constexpr int kAtQBytes = 2 * kAtQChunk, kAtStage = 4 * kAtKvChunk;      // a stage: keys, values
constexpr int kAtBars = kAtQBytes + kAtStages * kAtStage, kAtSmem = kAtBars + 1024 + 6144;
constexpr int kAtIssueWarp = 16, kAtLoadWarp = 17;

struct AtShared {
  uint64_t q_full, full[kAtStages], empty[kAtStages], s_full[2], p_full[2], o_full[2], o_free[2], al_full[4], done;
  uint32_t tmem_base;
  int gave_up;
  float met[2][2][kAtRows];       // by turns: what the threads of a row have found in their half of the keys
  // Factor of the sums before a tile.  Four tiles: scores of tile j + 4 come after the product of j + 2, and that after the sums of j.
  float al[4][kAtRows];
  float stat[2][kAtRows];         // maximum and sum of a row in the end
};
static_assert(sizeof(AtShared) <= 6144, "");

// Barrier of the two warps of 32 rows; whether any of their threads has failed.
__device__ __forceinline__ bool at_pair_failed(int id, bool failed) {
  uint32_t any;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
      "barrier.red.or.pred p, %2, 64, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(any) : "r"((uint32_t)failed), "r"(id) : "memory");
  return any != 0;
}

__global__ void __launch_bounds__(kAtTileThreads, 1)
attn_tile_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const __grid_constant__ AttnRowsArgs a,
                 const int* __restrict__ cu, int tiles, int tt) {
  using namespace sm100;
  extern __shared__ __align__(128) uint8_t atsm_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(atsm_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* kv = smem + kAtQBytes;
  AtShared* sh = reinterpret_cast<AtShared*>(smem + kAtBars);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (warp == kAtIssueWarp) tmem_alloc<512>(&sh->tmem_base);
  tc_fence_before();
  __syncthreads();                                     // the TMEM is this CTA's before the next kernel's CTAs come in
  tc_fence_after();
  chain_next();
  chain_wait(cu);
  AtTile T;
  const bool any = T.init(a, cu, tiles, tt);
  const int rows = any ? T.rows : 0, warps = any ? (rows + 31) / 32 : 1;  // groups of 32 rows
  if (threadIdx.x == 0) {
    mbar_init(&sh->q_full, 2 * warps);
    for (int i = 0; i < kAtStages; ++i) {
      mbar_init(&sh->full[i], 1);
      mbar_init(&sh->empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&sh->s_full[i], 1);
      mbar_init(&sh->p_full[i], 2 * warps);
      mbar_init(&sh->o_full[i], 1);
      mbar_init(&sh->o_free[i], 2 * warps);
    }
    for (int i = 0; i < 4; ++i) mbar_init(&sh->al_full[i], warps);
    mbar_init(&sh->done, warps);
    sh->gave_up = *(volatile int*)a.err;               // an earlier kernel already failed: do not wait on anything
    fence_barrier_init();
  }
  __syncthreads();
  const uint32_t tmem = sh->tmem_base;
  volatile int* gave_up = &sh->gave_up;
  const bool dead = *gave_up != 0;
  const int n_tiles = any && T.k1 > T.k0 ? (T.k1 - T.k0 + kAtTile - 1) / kAtTile : 0;
  const int kc = (a.d + 63) / 64, vc = (a.dv + 63) / 64;                // 64-column chunks of a key, of a value
  auto fail = [&]() {
    *gave_up = 1;
    atomicCAS(a.err, 0, kAfErr);
  };

  if (!any || dead) {
    // nothing was issued
  } else if (warp == kAtLoadWarp) {
    if (lane == 0) {
      for (int j = 0; j < n_tiles; ++j) {
        const int s = j % kAtStages, row = (int)T.base + T.k0 + j * kAtTile;    // rows past the tensor are zero-filled
        if (!mbar_wait(&sh->empty[s], ((j / kAtStages) & 1) ^ 1, gave_up)) {
          fail();
          break;
        }
        mbar_expect_tx(&sh->full[s], (kc + vc) * kAtKvChunk);
        uint8_t* st = kv + s * kAtStage;
        for (int c = 0; c < kc; ++c) tma_load_3d(st + c * kAtKvChunk, &tmK, &sh->full[s], c * 64, T.g, row);
        for (int c = 0; c < vc; ++c) tma_load_3d(st + (2 + c) * kAtKvChunk, &tmV, &sh->full[s], c * 64, T.g, row);
      }
    }
  } else if (warp == kAtIssueWarp) {
    constexpr uint32_t idesc_s = make_idesc_bf16(128, kAtTile, false, false);
    const uint32_t idesc_o = make_idesc_bf16(128, a.dv, false, true);
    const uint32_t e = elect_one(), tm = __reduce_or_sync(0xffffffffu, tmem);
    const uint64_t q_desc = make_smem_desc(smem_u32(smem), 16, 1024), k_desc = make_smem_desc(smem_u32(kv), 16, 1024);
    const uint64_t v_desc = make_smem_desc(smem_u32(kv) + 2 * kAtKvChunk, kAtKvChunk, 1024);
    const int ksteps = a.d / 16;
    // The scores of a tile go over the parts of the one two before: those products were issued earlier, and are taken in order.
    auto scores = [&](int j) -> bool {
      const int s = j % kAtStages;
      if (!mbar_wait_warp(&sh->full[s], (j / kAtStages) & 1, gave_up)) return false;
      tc_fence_after();
      const uint64_t kd = k_desc + s * (kAtStage >> 4);
      const uint32_t dst = tm + (j & 1) * 128;
      if (ksteps == 8) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_bf16_warp(e, dst, q_desc + (((k >> 2) * kAtQChunk + (k & 3) * 32) >> 4), kd + (((k >> 2) * kAtKvChunk + (k & 3) * 32) >> 4),
                         idesc_s, k != 0);
      } else {
#pragma unroll 1
        for (int k = 0; k < ksteps; ++k)
          umma_bf16_warp(e, dst, q_desc + (((k >> 2) * kAtQChunk + (k & 3) * 32) >> 4), kd + (((k >> 2) * kAtKvChunk + (k & 3) * 32) >> 4),
                         idesc_s, k != 0);
      }
      umma_commit_warp(e, &sh->s_full[j & 1]);
      return true;
    };
    bool ok = n_tiles == 0 || (mbar_wait_warp(&sh->q_full, 0, gave_up) && scores(0));
    if (ok && n_tiles > 1) ok = scores(1);
    for (int j = 0; j < n_tiles && ok; ++j) {
      const int s = j % kAtStages, b = j & 1;
      const uint32_t ph = (j >> 1) & 1;
      ok = mbar_wait_warp(&sh->p_full[b], ph, gave_up) && (j < 2 || mbar_wait_warp(&sh->o_free[b], ph ^ 1, gave_up));
      if (!ok) break;
      tc_fence_after();
      const uint64_t vd = v_desc + s * (kAtStage >> 4);
      const uint32_t dst = tm + 256 + b * 128, p = tm + b * 128;
#pragma unroll
      for (int x = 2; x >= 0; --x)
#pragma unroll
        for (int k = 0; k < kAtTile / 16; ++k)
          umma_bf16_ts_warp(e, dst, p + x * 32 + k * 8, vd + ((k * 2048) >> 4), idesc_o, x != 2 || k != 0);
      umma_commit_warp(e, &sh->empty[s]);
      umma_commit_warp(e, &sh->o_full[b]);
      if (j + 2 < n_tiles) ok = scores(j + 2);
    }
    if (!ok && e) fail();
  } else if ((warp & 3) < warps && warp < 8) {
    // ------------------------------- softmax -------------------------------
    const int quad = warp & 3, half = warp >> 2, row = quad * 32 + lane;
    const int m = min(row, rows - 1), tok = T.token(m), head = T.head(m);                   // rows past the end repeat the last
    {
      const __nv_bfloat16* q = reinterpret_cast<const __nv_bfloat16*>(a.q);
      const bool wide = a.ldq % 8 == 0 && (reinterpret_cast<uintptr_t>(q) & 15) == 0;
      const unsigned long long mine = reinterpret_cast<unsigned long long>(q + (size_t)tok * a.ldq + (size_t)head * a.d);
      if (wide) {                                      // sixteen lanes a row, each warp half of the rows
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
          const int r = half * 16 + i + (lane >> 4), piece = lane & 15, at = quad * 32 + r;
          const uint4* src = reinterpret_cast<const uint4*>(__shfl_sync(0xffffffffu, mine, r)) + piece;
          if (piece * 8 < kc * 64)
            *reinterpret_cast<uint4*>(smem + (piece >> 3) * kAtQChunk + at * 128 + (((piece ^ at) & 7) << 4)) =
                piece * 8 < a.d ? *src : make_uint4(0, 0, 0, 0);
        }
      } else {
#pragma unroll 4
        for (int i = 0; i < 32; ++i) {
          const int r = half * 16 + (i >> 1), word = (i & 1) * 32 + lane, at = quad * 32 + r, piece = word >> 2;
          const uint32_t* src = reinterpret_cast<const uint32_t*>(__shfl_sync(0xffffffffu, mine, r)) + word;
          if (word * 2 < kc * 64)
            *reinterpret_cast<uint32_t*>(smem + (piece >> 3) * kAtQChunk + at * 128 + (((piece ^ at) & 7) << 4) + (word & 3) * 4) =
                word * 2 < a.d ? *src : 0u;
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh->q_full);
    }
    const int end = a.len[tok], first = max(0, end - a.window);
    const bool bias = a.slopes != nullptr;
    const float slope = bias ? a.slopes[head] : 0.f;
    const uint32_t t_row = tmem + ((uint32_t)(quad * 32) << 16), t_s = t_row + half * kAtHalf, t_p = t_row + half * (kAtHalf / 2);
    float mx = -INFINITY, l = 0.f;
    bool failed = false;
    for (int j = 0; j < n_tiles; ++j) {
      const uint32_t turn = (j & 1) * 128;
      // this also says that the products of two tiles before have been made: they were issued earlier
      failed = !mbar_wait(&sh->s_full[j & 1], (j >> 1) & 1, gave_up);
      __syncwarp();
      tc_fence_after();
      uint32_t s[kAtHalf];
      tmem_ld_32x32(t_s + turn, s);
      tmem_ld_wait();
      const int key0 = T.k0 + j * kAtTile + half * kAtHalf;
#pragma unroll
      for (int i = 0; i < kAtHalf; ++i) s[i] = __float_as_uint(__uint_as_float(s[i]) * a.scale);
      if (bias) {
#pragma unroll
        for (int i = 0; i < kAtHalf; ++i)
          s[i] = __float_as_uint(fmaf(slope, (float)(key0 + i - (end - 1)), __uint_as_float(s[i])));
      }
      if (key0 + kAtHalf > min(T.len0, T.k1) || key0 < T.last_first) {
        const int lo = first - key0, hi = end - 1 - key0;
        uint32_t seen = hi < 0 ? 0u : 0xffffffffu >> (31 - min(hi, 31));
        if (lo > 0) seen = lo > 31 ? 0u : seen & (0xffffffffu << lo);
#pragma unroll
        for (int i = 0; i < kAtHalf; ++i)
          if (!(seen >> i & 1)) s[i] = 0xff800000u;    // -inf
      }
      float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < kAtHalf; i += 8)
#pragma unroll
        for (int x = 0; x < 4; ++x) m4[x] = fmax3(m4[x], __uint_as_float(s[i + 2 * x]), __uint_as_float(s[i + 2 * x + 1]));
      const float here = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
      sh->met[j & 1][half][row] = here;
      // both have read their scores too: the parts may go over them
      tc_fence_before();
      if (at_pair_failed(quad + 1, failed)) {
        failed = true;
        break;
      }
      tc_fence_after();
      const float now = fmaxf(mx, fmaxf(here, sh->met[j & 1][half ^ 1][row]));
      const float al = now == mx ? 1.f : expf(mx - now);                     // no key yet: nothing to rescale
      if (half == 0) {
        sh->al[j & 3][row] = al;
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh->al_full[j & 3]);
      }
      mx = now;
      l *= al;
      const float ref = mx == -INFINITY ? 0.f : mx;    // no key yet: all weights 0
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int c = 0; c < kAtHalf; c += 16) {
        uint32_t part[3][8];
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
          const float p0 = expf(__uint_as_float(s[c + i]) - ref), p1 = expf(__uint_as_float(s[c + i + 1]) - ref);
          sum[i & 2] += p0;
          sum[(i & 2) + 1] += p1;
          uint32_t p[3];
          cut_bf16(p0, p1, p);
#pragma unroll
          for (int x = 0; x < 3; ++x) part[x][i >> 1] = p[x];
        }
#pragma unroll
        for (int x = 0; x < 3; ++x) tmem_st_32x8(t_p + turn + x * 32 + c / 2, part[x]);
      }
      l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
      const int behind = T.k0 + (j + 1) * kAtTile - T.k1;
      if (behind > 0) {                                // rows past the range: 0 times what a former sequence left there must be 0
        const int s = j % kAtStages;
        failed = failed || !mbar_wait(&sh->full[s], (j / kAtStages) & 1, gave_up);
        uint8_t* left = kv + s * kAtStage + 2 * kAtKvChunk + (kAtTile - behind) * 128;
        for (int c = 0; c < vc; ++c)
          for (int p = (half * warps + quad) * 32 + lane; p < behind * 8; p += 64 * warps)
            *reinterpret_cast<uint4*>(left + c * kAtKvChunk + p * 16) = make_uint4(0, 0, 0, 0);
        fence_proxy_async_smem();
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh->p_full[j & 1]);
    }
    sh->met[n_tiles & 1][half][row] = l;
    if (at_pair_failed(quad + 1, failed)) {
      fail();
    } else if (half == 0) {
      sh->stat[0][row] = mx;
      sh->stat[1][row] = l + sh->met[n_tiles & 1][1][row];
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh->done);
    }
  } else if ((warp & 3) < warps && warp < 16) {
    // ------------------------------- sums -------------------------------
    const int quad = warp & 3, half = (warp - 8) >> 2, row = quad * 32 + lane;
    const uint32_t t_o = tmem + ((uint32_t)(quad * 32) << 16) + 256 + half * 64;
    const int mine = min(64, a.dv - half * 64);        // this thread's columns (none: not above 0)
    float acc[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) acc[i] = 0.f;
    bool failed = false;
    for (int j = 0; j < n_tiles; ++j) {
      failed = !mbar_wait_warp(&sh->al_full[j & 3], (j >> 2) & 1, gave_up) || !mbar_wait_warp(&sh->o_full[j & 1], (j >> 1) & 1, gave_up);
      if (failed) break;
      tc_fence_after();
      const float al = sh->al[j & 3][row];
#pragma unroll
      for (int c = 0; c < 64; c += 16) {
        if (c < mine) {
          uint32_t v[16];
          tmem_ld_32x16(t_o + (j & 1) * 128 + c, v);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) acc[c + i] = fmaf(acc[c + i], al, __uint_as_float(v[i]));
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh->o_free[j & 1]);
    }
    failed = failed || !mbar_wait_warp(&sh->done, 0, gave_up);
    if (at_pair_failed(quad + 5, failed)) {
      fail();
    } else {
      // Rows leave 32 columns at a time through the warp's own place in the stages, which nobody reads any more, so that a store
      // covers neighbouring columns.
      const int m = min(row, rows - 1);
      const float mx = sh->stat[0][row], l = sh->stat[1][row];
      float* stage = reinterpret_cast<float*>(kv) + (warp - 8) * 32 * 33;
      float f = 1.f, *part = nullptr;
      __nv_bfloat16* out = T.place(a, m, mx, l, f, part);
      if (row < rows && half == 0 && part != nullptr) {
        part[0] = mx;
        part[1] = l;
      }
      const unsigned long long to = part != nullptr ? reinterpret_cast<unsigned long long>(part + 2) : reinterpret_cast<unsigned long long>(out);
      const int n_rows = min(32, rows - quad * 32);
      float probe = l * 0.f;                           // NaN once a value is not finite
#pragma unroll
      for (int c0 = 0; c0 < 64; c0 += 32) {
        if (c0 < mine) {
          const int cols = min(32, mine - c0), c = half * 64 + c0;
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            probe = fmaf(acc[c0 + i], 0.f, probe);
            stage[lane * 33 + i] = acc[c0 + i] * f;
          }
          __syncwarp();
          if (part != nullptr) {
#pragma unroll 8
            for (int r = 0; r < n_rows; ++r) {
              float* dst = reinterpret_cast<float*>(__shfl_sync(0xffffffffu, to, r)) + c;
              if (lane < cols) dst[lane] = stage[r * 33 + lane];
            }
          } else {
#pragma unroll 4
            for (int r = 0; r < n_rows; r += 2) {      // two rows a store, two columns a lane
              const int rr = r + (lane >> 4), col = (lane & 15) * 2;
              __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(__shfl_sync(0xffffffffu, to, rr & 31)) + c + col;
              if (rr < n_rows && col < cols)
                *reinterpret_cast<__nv_bfloat162*>(dst) = __floats2bfloat162_rn(stage[rr * 33 + col], stage[rr * 33 + col + 1]);
            }
          }
          __syncwarp();
        }
      }
      // rows with values that are not finite, once both halves of them are written
      sh->met[0][half][row] = not_finite(probe) ? 1.f : 0.f;
      at_pair_failed(quad + 5, false);
      const bool odd_row = row < rows && half == 0 && sh->met[0][0][row] + sh->met[0][1][row] > 0.f;
      for (uint32_t odd = __ballot_sync(0xffffffffu, odd_row); odd != 0; odd &= odd - 1) at_row_alone(a, T, quad * 32 + __ffs(odd) - 1);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*gave_up && !dead && threadIdx.x == 0) {         // copies and products still in flight end before their memory goes away
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) {
    }
  }
  __syncthreads();
  if (warp == kAtIssueWarp) {
    tc_fence_after();
    tmem_dealloc<512>(tmem);
  }
}

// How a call runs on these kernels: tokens and CTAs of a tile, ranges of keys.  One sequence per `cu` entry, or one token
// each.  Ranges are of 128 keys at least.
struct AtPlan {
  bool fits, few;
  int tt, tiles, splits, range;
};
// Ranges of decoding rows.  A CTA draws 47 GB/s, all together 6.4 TB/s (136 of them), and two an SM are resident: full rounds of CTAs go at
// the second rate, the last one at what its CTAs draw; a round costs 1.5 us besides, a merge 3.5.  The bound of the lengths may be
// met by all rows, or by one where the mean is half of it: the sum of both decides.  Measured (us; ranges 1 / 2 / 3 / 4): 64 sequences of
// 2100 keys, 32 query heads on 8, 86 / 95 / 98 / 98; 48 of 2048 73 / 69 / 71 / 73; 24 of 3000 48 / 56 / 54 / 55; 8 of 4200, 16 on 8, 49 / 31 / 28 /
// 28 (5: 32); 10 of 2048, 32 on 32, 70 / 63 / 62 / 62; 40 of 64 to 4096, 16 on 4, 50 / 37 / 35 / 39; 16 of 100 in caches of 512 5 / 7 / 8 / 9.
static int at_ranges(long long ctas, long long most, double bytes_of_cta) {
  constexpr double kAll = 6.4e6, kOne = 47e3;          // bytes a us
  const long long resident = 2 * kNumSMs;
  int best = 1;
  double least = 1e30;
  for (int s = 1; s <= most; ++s) {
    const double b = bytes_of_cta / s;
    const long long n = ctas * s, rounds = (n - 1) / resident, last = n - rounds * resident;
    const double alike = rounds * (resident * b / kAll + 1.5) + std::max(last * b / kAll, b / kOne);
    const double varied = std::max(n * b / 2 / kAll, b / kOne);
    const double us = alike + varied + (s > 1 ? 7.0 : 0.0);
    if (us < least) {
      least = us;
      best = s;
    }
  }
  return best;
}
// Ranges of continued prompts.  A CTA an SM takes 1.5 us a tile of 64 keys and 5 beside them; the ranges' sums are written and read once
// at 3 TB/s, and their merge is a launch of 4.5 us.  Measured, us (ranges 1 / 2 / 3 / 4 / 6): 301 tokens of two sequences over 3000, 16 heads on
// 8 (48 CTAs), 74 / 50 / 42 / 60 / 52; 512 tokens over 4096, 32 on 8 (128), 100 / 130 / 138 / 148 / 161; 700 over 2000, 16 on 16 (96), 54 / 75 /
// 69 / 77 / 87; 17 over 3000, 32 on 8 (8), 71 / 44 / 34 / 28 / 24, with 18 20.
static int at_tile_ranges(long long ctas, long long most, int max_len, double bytes) {
  int best = 1;
  double least = 1e30;
  for (int s = 1; s <= most; ++s) {
    const long long rounds = (ctas * s + kNumSMs - 1) / kNumSMs, tiles = ((max_len + s - 1) / s + kAtTile - 1) / kAtTile;
    const double us = rounds * (tiles * 1.5 + 5) + (s > 1 ? 4.5 + bytes * s / 3e6 : 0.0);
    if (us < least) {
      least = us;
      best = s;
    }
  }
  return best;
}
static AtPlan at_plan(int n, int n_seq, int max_q, int H, int G, int d, int dv, int max_len, int window, bool is_bf16) {
  AtPlan p{};
  p.fits = is_bf16 && d % 16 == 0 && dv % 16 == 0 && d <= 128 && dv <= 128 && d > 0 && dv > 0;
  if (!p.fits) return p;
  const int rep = H / G, groups = (rep + kAtHeads - 1) / kAtHeads, nh = rep < kAtHeads ? rep : kAtHeads;
  const bool one = n_seq <= 0 || max_q <= 1;
  p.few = one || max_q * nh <= 16;
  p.tt = one ? 1 : (p.few ? 16 : kAtRows) / nh;
  p.tiles = one ? 1 : (max_q + p.tt - 1) / p.tt;
  const long long ctas = (long long)(one ? n : n_seq * p.tiles) * G * groups;
  if (window > 0 && max_len > window) max_len = window;
  max_len += p.tt - 1;                                  // a tile's rows see windows that start apart
  const long long most = std::min<long long>((max_len + 127) / 128, kArMaxSplits);
  long long s;
  if (p.few) {
    s = at_ranges(ctas, most, (double)max_len * (d + dv) * 2);
  } else {                                              // no more tiles than the tokens fill, and one a sequence that is not full
    const long long filled = std::min<long long>((long long)n_seq * p.tiles, n / p.tt + n_seq);
    s = at_tile_ranges(filled * G * groups, most, max_len, (double)n * H * (dv + 2) * 8);
  }
  p.splits = (int)s;
  p.range = ((max_len + p.splits - 1) / p.splits + 63) / 64 * 64;
  return p;
}

int make_tmap_bf16_2d(CUtensorMap* map, const void* ptr, uint64_t inner, uint64_t outer, uint64_t row_stride_bytes,
                      uint32_t box_inner, uint32_t box_outer);
int make_tmap_bf16_heads(CUtensorMap* map, const void* ptr, uint64_t dim, uint64_t heads, uint64_t rows, uint64_t row_stride_bytes,
                         uint32_t box_dim, uint32_t box_rows, uint64_t head_stride_bytes);

template <typename Kernel>
static int allow_smem(Kernel kern, int smem, bool& configured) {
  if (configured) return 0;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  configured = e == cudaSuccess;
  return (int)e;
}
static int launch_attn_cached(const AttnRowsArgs& a, const AtPlan& p, const int* cu, int n_seq, long long rows, cudaStream_t stream) {
  const int rep = a.H / a.G, nh = rep < kAtHeads ? rep : kAtHeads, groups = (rep + kAtHeads - 1) / kAtHeads;
  if (p.tt == 1) cu = nullptr;
  const dim3 grid(p.tt == 1 ? a.n : n_seq * p.tiles, a.G * groups, p.splits);
  if (grid.y > 65535) return -2;
  CUtensorMap tk, tv;
  const int box = p.few ? kAfKeys : kAtTile;
  int rc = make_tmap_bf16_heads(&tk, a.k, a.d, a.G, rows, (uint64_t)a.ldk * 2, 64, box, 0);
  if (!rc) rc = make_tmap_bf16_heads(&tv, a.v, a.dv, a.G, rows, (uint64_t)a.ldv * 2, 64, box, 0);
  if (rc) return rc;
  if (!p.few) {
    static bool tile = false;
    if ((rc = allow_smem(attn_tile_kernel, kAtSmem, tile)) != 0) return rc;
    launch_chained(attn_tile_kernel, grid, kAtTileThreads, kAtSmem, stream, tk, tv, a, cu, p.tiles, p.tt);
  } else {
    const bool full = a.d == 128 && a.dv == 128, small = p.tt * nh <= 8;
#define ELL_FEW(NB_, FULL_)                                                                                                   \
  if (small == (NB_ == 1) && full == FULL_) {                                                                                 \
    static bool ready = false;                                                                                                \
    if ((rc = allow_smem(attn_few_kernel<NB_, FULL_>, kAfSmem, ready)) != 0) return rc;                                       \
    launch_chained(attn_few_kernel<NB_, FULL_>, grid, kAtThreads, kAfSmem, stream, tk, tv, a, cu, p.tiles, p.tt);              \
  }
    ELL_FEW(1, true)
    ELL_FEW(1, false)
    ELL_FEW(2, true)
    ELL_FEW(2, false)
#undef ELL_FEW
  }
  if (a.splits > 1) launch_chained(attn_rows_merge_kernel<__nv_bfloat16>, dim3(a.n, a.H), kArThreads, 0, stream, a);
  return launch_status();
}

static int al_mt(int H) { return H > 16 ? 2 : 1; }

// Ranges per row of the latent kernel: one CTA an SM, at least one tile each.
static int attn_latent_splits(int n, int H, int max_len) {
  const long long ctas = (long long)n * ((H + 16 * al_mt(H) - 1) / (16 * al_mt(H)));
  long long s = kNumSMs / ctas;
  const long long most = (max_len + kAlKeys - 1) / kAlKeys;
  if (s > most) s = most;
  if (s > kArMaxSplits) s = kArMaxSplits;
  return s < 1 ? 1 : (int)s;
}

template <int MT>
static int launch_attn_latent(const AttnRowsArgs& a, long long rows, cudaStream_t stream) {
  CUtensorMap tk;
  const int rc = make_tmap_bf16_2d(&tk, a.k, (uint64_t)a.d, (uint64_t)rows, (uint64_t)a.ldk * 2, 64, kAlKeys);
  if (rc) return rc;
  const int bytes = al_bytes(a.d, MT);
  static int configured = 0;
  if (bytes > configured) {
    cudaError_t e = cudaFuncSetAttribute(attn_latent_kernel<MT>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return (int)e;
    configured = bytes;
  }
  launch_chained(attn_latent_kernel<MT>, dim3(a.n, (a.H + 16 * MT - 1) / (16 * MT), a.splits), kAlWarps * 32, bytes, stream, tk, a);
  if (a.splits > 1) launch_chained(attn_rows_merge_kernel<__nv_bfloat16>, dim3(a.n, a.H), kArThreads, 0, stream, a);
  return launch_status();
}

// Shapes of the mma kernel; everything else runs on attn_rows_kernel.
static bool attn_latent_fits(const void* k, int d, int dv, int ldq, int ldk, int H) {
  return aligned_to(k, 16) && d % 8 == 0 && dv % 8 == 0 && dv <= d && dv <= 8 * kAlWarps * kAlMaxNt && ldq % 8 == 0 && ldk % 8 == 0 &&
         H <= 65535 && al_bytes(d, al_mt(H)) <= 227 * 1024;
}

// Query heads a CTA takes.
static int ar_rep(int rep) { return rep <= 4 ? 4 : kArRep; }

// Ranges per row: enough CTAs to fill the GPU a few times, about 256 keys each at least.
static int attn_rows_splits(int n, int H, int G, int max_len) {
  const int rep = H / G;
  const long long ctas = (long long)n * G * ((rep + ar_rep(rep) - 1) / ar_rep(rep));
  long long s = (4LL * kNumSMs + ctas - 1) / ctas;
  const long long most = (max_len + 255) / 256;
  if (s > most) s = most;
  if (s > kArMaxSplits) s = kArMaxSplits;
  return s < 1 ? 1 : (int)s;
}

template <typename T, int KT, int REP, bool VEC>
static int launch_attn_rows_kt(const AttnRowsArgs& a, dim3 grid, cudaStream_t stream) {
  const int bytes = ar_layout(a.d, a.dv, sizeof(T), KT, REP).bytes;
  auto kern = attn_rows_kernel<T, KT, REP, VEC>;
  static int configured = 0;
  if (bytes > configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return (int)e;
    configured = bytes;
  }
  launch_chained(kern, grid, kArThreads, bytes, stream, a);
  if (a.splits > 1) launch_chained(attn_rows_merge_kernel<T>, dim3(a.n, a.H), kArThreads, 0, stream, a);
  return launch_status();
}

template <typename T, int REP>
static int launch_attn_rows(const AttnRowsArgs& a, dim3 grid, bool vec, cudaStream_t stream) {
  const bool small = ar_layout(a.d, a.dv, sizeof(T), 32, REP).bytes > 160 * 1024;      // very wide fp32 heads: short tiles
  if (small) return vec ? launch_attn_rows_kt<T, 16, REP, true>(a, grid, stream) : launch_attn_rows_kt<T, 16, REP, false>(a, grid, stream);
  return vec ? launch_attn_rows_kt<T, 32, REP, true>(a, grid, stream) : launch_attn_rows_kt<T, 32, REP, false>(a, grid, stream);
}

}  // namespace ell

using namespace ell;

// Scratch floats a call needs (0: none).  The sizes are those of ell_attn_rows.
ELL_API long long ell_attn_rows_scratch(int n, int H, int G, int d, int dv, int max_len, int window, int n_seq, int max_q,
                                        int is_bf16) {
  const AtPlan p = at_plan(n, n_seq, max_q, H, G, d, dv, max_len, window, is_bf16);
  const int most = window > 0 && max_len > window ? window : max_len, rows = attn_rows_splits(n, H, G, most);
  const int s = p.fits && p.splits > rows ? p.splits : rows;       // enough for either kernel
  return s == 1 ? 0 : (long long)n * H * s * (dv + 2);
}

// Rows of ldq / ldk / ldv elements; max_len bounds len[] (it sets the number of ranges, longer rows would be cut).
// window: keys a row sees (<= 0: all).  gate: rows of ldg elements of the activation type, or null.
// cu [n_seq + 1] (or null): rows cu[i] .. cu[i + 1] - 1 are consecutive tokens of one sequence, with one base and lengths that
// grow by one; max_q bounds their number.  kv_rows: rows of k and v.
ELL_API int ell_attn_rows(const void* q, const void* k, const void* v, void* out, float* part, const int* base,
                          const int* len, const float* sink, const float* slopes, const void* gate, int n, int H, int G,
                          int d, int dv, int ldq, int ldk, int ldv, int ldg, int max_len, int window, float scale,
                          const int* cu, int n_seq, int max_q, long long kv_rows, int is_bf16, int* err, cudaStream_t stream) {
  if (n <= 0) return 0;
  if (H % G || dv > 8 * kArThreads || H > 65535) return -2;
  const AtPlan p = at_plan(n, cu != nullptr ? n_seq : 0, max_q, H, G, d, dv, max_len, window, is_bf16);
  if (window <= 0) window = 0x7fffffff;
  if (max_len > window) max_len = window;
  AttnRowsArgs a{q, k, v, out, part, base, len, sink, slopes, n, H, G, d, dv, ldq, ldk, ldv, 1, 0, scale, window, gate, ldg, err, 0};
  const int esz = is_bf16 ? 2 : 4;
  const bool vec = (d * esz) % 16 == 0 && (dv * esz) % 16 == 0 && (ldk * esz) % 16 == 0 && (ldv * esz) % 16 == 0 &&
                   aligned_to(k, 16) && aligned_to(v, 16);
  if (p.fits && vec && ldq % 2 == 0 && aligned_to(q, 4) && kv_rows <= 0x7fffffff) {
    a.splits = p.splits;
    a.range = p.range;
    a.all_ranges = p.tt > 1;
    if (a.splits > 1 && part == nullptr) return -2;
    return launch_attn_cached(a, p, cu, n_seq, kv_rows, stream);
  }
  a.splits = attn_rows_splits(n, H, G, max_len);
  a.range = ((max_len + a.splits - 1) / a.splits + 63) / 64 * 64;
  if (a.splits > 1 && part == nullptr) return -2;
  const int rep = H / G, per = ar_rep(rep);
  dim3 grid(n, G * ((rep + per - 1) / per), a.splits);
  if (ar_layout(d, dv, esz, 16, per).bytes > 227 * 1024) return -2;
  if (is_bf16)
    return per == 4 ? launch_attn_rows<__nv_bfloat16, 4>(a, grid, vec, stream) : launch_attn_rows<__nv_bfloat16, 8>(a, grid, vec, stream);
  return per == 4 ? launch_attn_rows<float, 4>(a, grid, vec, stream) : launch_attn_rows<float, 8>(a, grid, vec, stream);
}

// Latent attention: q [n, H, d] (rows of ldq), one key row [d] per position (`rows` rows of ldk) whose first dv columns are
// the value -> out [n, H, dv].  bf16 shapes the mma kernel takes run there, others on attn_rows.
ELL_API long long ell_attn_latent_scratch(const void* k, int n, int H, int d, int dv, int ldq, int ldk, int max_len, int window, int is_bf16) {
  if (window > 0 && max_len > window) max_len = window;
  if (!(is_bf16 && attn_latent_fits(k, d, dv, ldq, ldk, H))) return ell_attn_rows_scratch(n, H, 1, d, dv, max_len, window, 0, 1, is_bf16);
  const int s = attn_latent_splits(n, H, max_len);
  return s == 1 ? 0 : (long long)n * H * s * (dv + 2);
}

ELL_API int ell_attn_latent(const void* q, const void* k, void* out, float* part, const int* base, const int* len,
                            const void* gate, int n, int H, int d, int dv, int ldq, int ldk, int ldg, int max_len, int window,
                            long long rows, float scale, int is_bf16, int* err, cudaStream_t stream) {
  if (n <= 0) return 0;
  if (!(is_bf16 && attn_latent_fits(k, d, dv, ldq, ldk, H)))
    return ell_attn_rows(q, k, k, out, part, base, len, nullptr, nullptr, gate, n, H, 1, d, dv, ldq, ldk, ldk, ldg, max_len,
                         window, scale, nullptr, 0, 1, rows, is_bf16, err, stream);
  if (!aligned_to(q, 16) || !aligned_to(k, 16) || !aligned_to(out, 16) || rows > 0x7fffffff) return -2;
  if (window <= 0) window = 0x7fffffff;
  if (max_len > window) max_len = window;
  AttnRowsArgs a{q, k, k, out, part, base, len, nullptr, nullptr, n, H, 1, d, dv, ldq, ldk, ldk, 1, 0, scale, window, gate, ldg, err, 0};
  a.splits = attn_latent_splits(n, H, max_len);
  a.range = ((max_len + a.splits - 1) / a.splits + kAlKeys - 1) / kAlKeys * kAlKeys;
  if (a.splits > 1 && part == nullptr) return -2;
  return al_mt(H) == 1 ? launch_attn_latent<1>(a, rows, stream) : launch_attn_latent<2>(a, rows, stream);
}
