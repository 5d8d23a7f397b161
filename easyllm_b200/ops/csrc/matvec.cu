// y = x · Wᵀ for a few rows of x (decoding) and for row lengths the TMA-fed GEMM cannot take: bound by the weight bytes.
//
// bf16: a warp multiplies 16 rows of W with up to 16 rows of x on mma.sync m16n8k16 (the products are few, the point is
// to keep the instruction count far below the load rate): a thread loads 8 consecutive k of a row with one 16-byte load
// and feeds them to two instructions, in an order of k that is the same for both operands.  The warps of a CTA split K.
// fp32, and shapes without 16-byte rows: a warp computes NW rows of W against MR rows of x, lanes striding over K, fp32
// fused multiply-adds, one shuffle reduction per result.
// Optional bias, tanh, fp32 output, or accumulation into an fp32 matrix; a batch of equally shaped products in grid.z.
#include "vec.cuh"

namespace ell {

constexpr int kMvWarps = 8;

struct MatvecArgs {
  const void *x, *w, *bias;
  void* out;
  long long xb, wb, ob;       // batch strides in elements
  int M, N, K, ldx, ldo;
  int out_f32, accumulate, act_tanh, ks;
};

template <typename T, int MR, int NW, bool VEC>
__global__ void __launch_bounds__(kMvWarps * 32) matvec_kernel(const MatvecArgs a) {
  chain_enter();
  __shared__ float red[kMvWarps][NW * MR];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ks = a.ks, part = warp % ks, n0 = (blockIdx.x * (kMvWarps / ks) + warp / ks) * NW, m0 = blockIdx.y * MR;
  const T* x = reinterpret_cast<const T*>(a.x) + blockIdx.z * a.xb + (size_t)m0 * a.ldx;
  const T* w = reinterpret_cast<const T*>(a.w) + blockIdx.z * a.wb + (size_t)n0 * a.K;
  float acc[NW][MR];
#pragma unroll
  for (int i = 0; i < NW; ++i)
#pragma unroll
    for (int m = 0; m < MR; ++m) acc[i][m] = 0.f;
  if (n0 < a.N) {
#pragma unroll 2
    for (int k = (part * 32 + lane) * 8; k < a.K; k += ks * 256) {
      float wf[NW][8];
#pragma unroll
      for (int i = 0; i < NW; ++i) {
        if (VEC && n0 + i < a.N) {
          load_v<8>(w + (size_t)i * a.K + k, wf[i]);
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) wf[i][j] = n0 + i < a.N && k + j < a.K ? to_f<T>(w[(size_t)i * a.K + k + j]) : 0.f;
        }
      }
#pragma unroll
      for (int m = 0; m < MR; ++m) {
        float xf[8];
        if (VEC && m0 + m < a.M) {
          load_v<8>(x + (size_t)m * a.ldx + k, xf);
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) xf[j] = m0 + m < a.M && k + j < a.K ? to_f<T>(x[(size_t)m * a.ldx + k + j]) : 0.f;
        }
#pragma unroll
        for (int i = 0; i < NW; ++i)
#pragma unroll
          for (int j = 0; j < 8; ++j) acc[i][m] = fmaf(wf[i][j], xf[j], acc[i][m]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < NW; ++i)
#pragma unroll
    for (int m = 0; m < MR; ++m) {
      const float v = warp_sum(acc[i][m]);
      if (lane == 0) red[warp][i * MR + m] = v;
    }
  __syncthreads();
  if (part != 0 || n0 >= a.N) return;
  for (int e = lane; e < NW * MR; e += 32) {
    const int i = e / MR, m = e % MR, n = n0 + i;
    if (n >= a.N || m0 + m >= a.M) continue;
    float v = 0.f;
    for (int p = 0; p < ks; ++p) v += red[warp + p][e];
    if (a.bias != nullptr) v += to_f<T>(reinterpret_cast<const T*>(a.bias)[n]);
    if (a.act_tanh) v = tanhf(v);
    const size_t o = blockIdx.z * a.ob + (size_t)(m0 + m) * a.ldo + n;
    if (a.accumulate) reinterpret_cast<float*>(a.out)[o] += v;
    else if (a.out_f32) reinterpret_cast<float*>(a.out)[o] = v;
    else reinterpret_cast<T*>(a.out)[o] = from_f<T>(v);
  }
}

__device__ __forceinline__ void mma_16816(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// MT tiles of 8 rows of x (from row blockIdx.y * 8 MT on).  Rows of W and of x past the end are clamped (their results are dropped); k past the end is
// clamped too, with x taken as zero.
template <int MT>
__global__ void __launch_bounds__(kMvWarps * 32) matvec_mma_kernel(const MatvecArgs a) {
  __shared__ float red[kMvWarps][16][8 * MT + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int ks = a.ks, part = warp % ks, n0 = (blockIdx.x * (kMvWarps / ks) + warp / ks) * 16;
  const int m0 = blockIdx.y * 8 * MT, M = a.M - m0;
  const __nv_bfloat16* x = reinterpret_cast<const __nv_bfloat16*>(a.x) + blockIdx.z * a.xb + (size_t)m0 * a.ldx;
  const __nv_bfloat16* w = reinterpret_cast<const __nv_bfloat16*>(a.w) + blockIdx.z * a.wb;
  const __nv_bfloat16* w0 = w + (size_t)min(n0 + g, a.N - 1) * a.K;
  const __nv_bfloat16* w1 = w + (size_t)min(n0 + g + 8, a.N - 1) * a.K;
  chain_next();
  {
    // the CTA's rows of W come into L2 while the kernel before this one ends, a row (16-byte pieces) a thread
    const int first = blockIdx.x * (kMvWarps / ks) * 16, rows = min(kMvWarps / ks * 16, a.N - first);
    if (threadIdx.x < rows && blockIdx.y == 0)
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(w + (size_t)(first + threadIdx.x) * a.K), "r"(a.K * 2)
                   : "memory");
  }
  chain_wait();
  const __nv_bfloat16* xr[MT];
#pragma unroll
  for (int m = 0; m < MT; ++m) xr[m] = x + (size_t)min(m * 8 + g, M - 1) * a.ldx;
  float c0[MT][4], c1[MT][4];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int i = 0; i < 4; ++i) c0[m][i] = c1[m][i] = 0.f;
  constexpr int U = 4;
  const int nkb = (a.K + 31) / 32;
  for (int kb = part; kb < nkb; kb += ks * U) {
    uint4 wa[U], wb[U], xv[U][MT];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = (kb + u * ks) * 32 + t * 8;
      const bool in = k < a.K;
      const int kc = in ? k : 0;
      wa[u] = *reinterpret_cast<const uint4*>(w0 + kc);
      wb[u] = *reinterpret_cast<const uint4*>(w1 + kc);
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        xv[u][m] = *reinterpret_cast<const uint4*>(xr[m] + kc);
        if (!in) xv[u][m] = make_uint4(0, 0, 0, 0);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        mma_16816(c0[m], wa[u].x, wb[u].x, wa[u].y, wb[u].y, xv[u][m].x, xv[u][m].y);
        mma_16816(c1[m], wa[u].z, wb[u].z, wa[u].w, wb[u].w, xv[u][m].z, xv[u][m].w);
      }
  }
#pragma unroll
  for (int m = 0; m < MT; ++m) {
    red[warp][g][m * 8 + 2 * t] = c0[m][0] + c1[m][0];
    red[warp][g][m * 8 + 2 * t + 1] = c0[m][1] + c1[m][1];
    red[warp][g + 8][m * 8 + 2 * t] = c0[m][2] + c1[m][2];
    red[warp][g + 8][m * 8 + 2 * t + 1] = c0[m][3] + c1[m][3];
  }
  __syncthreads();
  const int rows = (kMvWarps / ks) * 16;
  for (int e = threadIdx.x; e < rows * 8 * MT; e += kMvWarps * 32) {
    const int r = e % rows, m = e / rows, n = blockIdx.x * rows + r;
    if (n >= a.N || m >= M) continue;
    float v = 0.f;
    for (int p = 0; p < ks; ++p) v += red[(r >> 4) * ks + p][r & 15][m];
    if (a.bias != nullptr) v += __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(a.bias)[n]);
    if (a.act_tanh) v = tanhf(v);
    const size_t o = blockIdx.z * a.ob + (size_t)(m0 + m) * a.ldo + n;
    if (a.accumulate) reinterpret_cast<float*>(a.out)[o] += v;
    else if (a.out_f32) reinterpret_cast<float*>(a.out)[o] = v;
    else reinterpret_cast<__nv_bfloat16*>(a.out)[o] = __float2bfloat16_rn(v);
  }
}

static int launch_matvec_mma(MatvecArgs a, int batch, cudaStream_t stream) {
  const int nkb = (a.K + 31) / 32, tiles = (a.N + 15) / 16;
  a.ks = kMvWarps;
  while (a.ks > 1 && (nkb < 4 * a.ks || (long long)tiles * batch * ((a.M + 15) / 16) * a.ks > 64LL * kNumSMs)) a.ks /= 2;
  const int per = kMvWarps / a.ks;
  dim3 grid((tiles + per - 1) / per, (a.M + 15) / 16, batch);
  if (grid.y > 65535) return -2;
  if (a.M <= 8) launch_chained(matvec_mma_kernel<1>, grid, kMvWarps * 32, 0, stream, a);
  else launch_chained(matvec_mma_kernel<2>, grid, kMvWarps * 32, 0, stream, a);
  return launch_status();
}

template <typename T, int MR, int NW>
int launch_matvec(MatvecArgs a, int batch, bool vec, cudaStream_t stream) {
  const long long warps = (long long)((a.N + NW - 1) / NW) * ((a.M + MR - 1) / MR) * batch;
  a.ks = 1;
  while (a.ks < kMvWarps && warps * a.ks < 12LL * kNumSMs && a.K >= 512 * a.ks) a.ks *= 2;
  const int per = kMvWarps / a.ks;
  dim3 grid(((a.N + NW - 1) / NW + per - 1) / per, (a.M + MR - 1) / MR, batch);
  if (grid.y > 65535) return -2;
  if (vec) launch_chained(matvec_kernel<T, MR, NW, true>, grid, kMvWarps * 32, 0, stream, a);
  else launch_chained(matvec_kernel<T, MR, NW, false>, grid, kMvWarps * 32, 0, stream, a);
  return launch_status();
}

template <typename T>
int dispatch_matvec(const MatvecArgs& a, int batch, bool vec, cudaStream_t stream) {
  if (a.M == 1) return launch_matvec<T, 1, 2>(a, batch, vec, stream);
  if (a.M == 2) return launch_matvec<T, 2, 2>(a, batch, vec, stream);
  if (a.M <= 4) return launch_matvec<T, 4, 2>(a, batch, vec, stream);
  return launch_matvec<T, 8, 4>(a, batch, vec, stream);
}

// ---- mixture of experts: routing, and the per-token products of a few tokens -----------------------
// One warp per token: the `top` largest router logits (ties: the lower index); scores sigmoid(z), or the softmax over the
// chosen logits.  bias [E] (or null) is added to the logits first.
__global__ void moe_route_kernel(const float* __restrict__ z, const float* __restrict__ bias, int* __restrict__ idx,
                                 float* __restrict__ w, int n, int E, int top, int ldz, int softmax) {
  chain_enter(z, bias, idx, w);
  const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (t >= n) return;
  const float* row = z + (size_t)t * ldz;
  uint32_t taken = 0;                                  // bit i: expert 32 i + lane
  float largest = 0.f, sum = 0.f;
  for (int k = 0; k < top; ++k) {
    float best = -INFINITY;
    int be = 0x7fffffff;
    for (int i = 0; 32 * i + lane < E; ++i)
      if (!(taken >> i & 1)) {
        const float v = row[32 * i + lane] + (bias != nullptr ? bias[32 * i + lane] : 0.f);
        if (v > best || be == 0x7fffffff) {
          best = v;
          be = 32 * i + lane;
        }
      }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oe = __shfl_xor_sync(0xffffffffu, be, o);
      if (oe != 0x7fffffff && (be == 0x7fffffff || ov > best || (ov == best && oe < be))) {
        best = ov;
        be = oe;
      }
    }
    if ((be & 31) == lane) taken |= 1u << (be >> 5);
    if (lane == 0) {
      if (k == 0) largest = best;
      const float e = softmax ? expf(best - largest) : sigmoid_f(best);
      sum += e;
      idx[t * top + k] = be;
      w[t * top + k] = e;
    }
  }
  if (softmax && lane == 0)
    for (int k = 0; k < top; ++k) w[t * top + k] /= sum;
}

// Router product and routing in one launch, bf16, up to 16 choices and 64 rows of W (experts first, then what else is wanted of the logits): 16 tokens
// a CTA, its warps split K as in matvec_mma_kernel.  The tiled product pads N to 128 and so filled 30 SMs with 3777 tokens of 2048:
// 14 us and 5.5 more for the routing, now 7; 64 tokens 8 and 3, now 5.5.
// The routing of moe_route_kernel for half a warp and up to 64 experts and 16 choices: lane k keeps choice k.
__device__ __forceinline__ void route_half(const float* row, const float* __restrict__ bias, int* __restrict__ idx, float* __restrict__ w,
                                           int E, int top, int softmax, int lane, uint32_t lanes) {
  float v[4], chosen = 0.f, largest = 0.f, sum = 0.f;
  int expert = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = i * 16 + lane < E ? row[i * 16 + lane] + (bias != nullptr ? bias[i * 16 + lane] : 0.f) : 0.f;
  uint32_t taken = 0;                                  // bit i: expert 16 i + lane
  for (int k = 0; k < top; ++k) {
    float best = -INFINITY;
    int be = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (i * 16 + lane < E && !(taken >> i & 1) && (v[i] > best || be == 0x7fffffff)) {
        best = v[i];
        be = i * 16 + lane;
      }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(lanes, best, o);
      const int oe = __shfl_xor_sync(lanes, be, o);
      if (oe != 0x7fffffff && (be == 0x7fffffff || ov > best || (ov == best && oe < be))) {
        best = ov;
        be = oe;
      }
    }
    if ((be & 15) == lane) taken |= 1u << (be >> 4);
    if (k == 0) largest = best;
    if (k == lane) {
      chosen = best;
      expert = be;
    }
  }
  float e = softmax ? expf(chosen - largest) : sigmoid_f(chosen);
  if (softmax) {
    for (int k = 0; k < top; ++k) sum += __shfl_sync(lanes, e, k, 16);
    e /= sum;
  }
  if (lane < top) {
    idx[lane] = expert;
    w[lane] = e;
  }
}

template <int NT>
__global__ void __launch_bounds__(kMvWarps * 32) moe_router_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                                                                    const float* __restrict__ bias, float* __restrict__ z,
                                                                    int* __restrict__ idx, float* __restrict__ score, int n, int N, int K,
                                                                    int ldx, int ldz, int E, int top, int softmax) {
  __shared__ float red[kMvWarps][16][8 * NT + 1];
  __shared__ float logits[16][8 * NT];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, t0 = blockIdx.x * 16;
  chain_next();
  if (blockIdx.x == 0 && threadIdx.x < N)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(w + (size_t)threadIdx.x * K), "r"(K * 2) : "memory");
  chain_wait(x, w, bias, z, idx, score);
  const __nv_bfloat16 *x0 = x + (size_t)min(t0 + g, n - 1) * ldx, *x1 = x + (size_t)min(t0 + g + 8, n - 1) * ldx;
  float c[NT][4];
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) c[i][j] = 0.f;
  constexpr int U = NT > 4 ? 2 : 4;
  for (int kb = warp; kb * 32 < K; kb += kMvWarps * U) {
    uint4 xa[U], xb[U], wv[U][NT];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = (kb + u * kMvWarps) * 32 + t * 8, kc = k < K ? k : 0;
      xa[u] = *reinterpret_cast<const uint4*>(x0 + kc);
      xb[u] = *reinterpret_cast<const uint4*>(x1 + kc);
      if (k >= K) xa[u] = xb[u] = make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int i = 0; i < NT; ++i) wv[u][i] = *reinterpret_cast<const uint4*>(w + (size_t)min(i * 8 + g, N - 1) * K + kc);
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        mma_16816(c[i], xa[u].x, xb[u].x, xa[u].y, xb[u].y, wv[u][i].x, wv[u][i].y);
        mma_16816(c[i], xa[u].z, xb[u].z, xa[u].w, xb[u].w, wv[u][i].z, wv[u][i].w);
      }
  }
#pragma unroll
  for (int i = 0; i < NT; ++i) {
    red[warp][g][i * 8 + 2 * t] = c[i][0];
    red[warp][g][i * 8 + 2 * t + 1] = c[i][1];
    red[warp][g + 8][i * 8 + 2 * t] = c[i][2];
    red[warp][g + 8][i * 8 + 2 * t + 1] = c[i][3];
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 16 * 8 * NT; e += kMvWarps * 32) {
    const int m = e / (8 * NT), i = e % (8 * NT);
    float v = 0.f;
#pragma unroll
    for (int p = 0; p < kMvWarps; ++p) v += red[p][m][i];
    logits[m][i] = v;
    if (i < N && t0 + m < n) z[(size_t)(t0 + m) * ldz + i] = v;
  }
  __syncthreads();
  const int m = warp * 2 + (lane >> 4);
  if (t0 + m < n)
    route_half(logits[m], bias, idx + (size_t)(t0 + m) * top, score + (size_t)(t0 + m) * top, E, top, softmax, lane & 15,
               lane < 16 ? 0xffffu : 0xffff0000u);
}

// For slot = token * top + k, a warp multiplies two weight rows of expert e = idx[slot] with the token:
//   GLU false  hidden units f0, f0 + 1 of up [E, F, W]:  hid[slot][f] = (w_slot relu(up_e[f] . h))^2
//   GLU true   the gate and up rows of one hidden unit of [E, 2 F, W], which alternate in blocks of `block` rows:
//              hid[slot][f] = w_slot silu(gate_e[f] . h) (up_e[f] . h)
template <typename T, bool VEC, bool GLU>
__global__ void __launch_bounds__(256) moe_up_kernel(const T* __restrict__ h, const T* __restrict__ up,
                                                     const int* __restrict__ idx, const float* __restrict__ wgt,
                                                     T* __restrict__ hid, int top, int F, int W, int block) {
  chain_enter(h, up, idx, wgt, hid);
  const int slot = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int f0 = (blockIdx.x * 8 + warp) * (GLU ? 1 : 2);
  if (f0 >= F) return;
  const T* x = h + (size_t)(slot / top) * W;
  const T* u0 = GLU ? up + ((size_t)idx[slot] * 2 * F + (size_t)(f0 / block) * 2 * block + f0 % block) * W
                    : up + ((size_t)idx[slot] * F + f0) * W;
  const bool two = GLU || f0 + 1 < F;
  const size_t second = GLU ? (size_t)block * W : (two ? W : 0);
  float a0 = 0.f, a1 = 0.f;
#pragma unroll 2
  for (int k = lane * 8; k < W; k += 256) {
    float xf[8], w0[8], w1[8];
    if (VEC) {
      load_v<8>(x + k, xf);
      load_v<8>(u0 + k, w0);
      load_v<8>(u0 + second + k, w1);
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const bool in = k + j < W;
        xf[j] = in ? to_f<T>(x[k + j]) : 0.f;
        w0[j] = in ? to_f<T>(u0[k + j]) : 0.f;
        w1[j] = in ? to_f<T>(u0[second + k + j]) : 0.f;
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      a0 = fmaf(xf[j], w0[j], a0);
      a1 = fmaf(xf[j], w1[j], a1);
    }
  }
  a0 = warp_sum(a0);
  a1 = warp_sum(a1);
  if (lane == 0) {
    const float s = wgt[slot];
    if (GLU) {
      hid[(size_t)slot * F + f0] = from_f<T>(s * silu_f(a0) * a1);
      return;
    }
    a0 = s * fmaxf(a0, 0.f);
    a1 = s * fmaxf(a1, 0.f);
    hid[(size_t)slot * F + f0] = from_f<T>(a0 * a0);
    if (two) hid[(size_t)slot * F + f0 + 1] = from_f<T>(a1 * a1);
  }
}

// acc[token][n] += sum over the token's experts of down_e[n] . hid; a warp owns two outputs of one token.
template <typename T, bool VEC>
__global__ void __launch_bounds__(256) moe_down_kernel(const T* __restrict__ hid, const T* __restrict__ down,
                                                       const int* __restrict__ idx, float* __restrict__ acc, int top, int F,
                                                       int W) {
  chain_enter(hid, down, idx, acc);
  const int t = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = (blockIdx.x * 8 + warp) * 2;
  if (n0 >= W) return;
  const bool two = n0 + 1 < W;
  float a0 = 0.f, a1 = 0.f;
  for (int s = 0; s < top; ++s) {
    const int slot = t * top + s;
    const T* x = hid + (size_t)slot * F;
    const T* d0 = down + ((size_t)idx[slot] * W + n0) * F;
#pragma unroll 2
    for (int k = lane * 8; k < F; k += 256) {
      float xf[8], w0[8], w1[8];
      if (VEC) {
        load_v<8>(x + k, xf);
        load_v<8>(d0 + k, w0);
        load_v<8>(d0 + (two ? F : 0) + k, w1);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const bool in = k + j < F;
          xf[j] = in ? to_f<T>(x[k + j]) : 0.f;
          w0[j] = in ? to_f<T>(d0[k + j]) : 0.f;
          w1[j] = in ? to_f<T>(d0[(two ? F : 0) + k + j]) : 0.f;
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        a0 = fmaf(xf[j], w0[j], a0);
        a1 = fmaf(xf[j], w1[j], a1);
      }
    }
  }
  a0 = warp_sum(a0);
  a1 = warp_sum(a1);
  if (lane == 0) {
    acc[(size_t)t * W + n0] += a0;
    if (two) acc[(size_t)t * W + n0 + 1] += a1;
  }
}

// ---- mixture of experts: rows sorted by expert for the grouped GEMM ---------------------------------
// Row plan and gathered rows in one launch.  Every expert's rows start at a multiple of 128, in the order of their slots (slot = token *
// top + k); tile_expert[i] is the expert of row tile i, *n_tiles their number, pos[slot] the row of a slot, row_scale[row] its score
// (rows of the padding: 0), xs[pos[slot]] = h[token].
// A CTA takes a range of slots and counts for itself, over all slots, the rows of every expert and those before its range: reading the
// indexes up to 296 times (30 kB for 3777 tokens, top 2) costs less than a plan made by one CTA and a launch that waits for it.  3777
// tokens of 2048: 20 us in two launches -> 11.5; 64 tokens 6.6 -> 4.6.
constexpr int kGatherThreads = 512;
__global__ void __launch_bounds__(kGatherThreads) moe_gather_kernel(const uint4* __restrict__ h, uint4* __restrict__ xs,
                                                                     const int* __restrict__ idx, const float* __restrict__ wgt,
                                                                     int* __restrict__ pos, float* __restrict__ row_scale,
                                                                     int* __restrict__ tile_expert, int* __restrict__ n_tiles, int slots,
                                                                     int top, int E, int wv) {
  __shared__ int total[1024], next[1024], first[1024], row[kGatherThreads];
  chain_enter(h, xs, idx, wgt, pos, row_scale, tile_expert, n_tiles);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int s0 = (int)((long long)slots * blockIdx.x / gridDim.x), s1 = (int)((long long)slots * (blockIdx.x + 1) / gridDim.x);
  for (int e = threadIdx.x; e < E; e += kGatherThreads) total[e] = next[e] = 0;
  __syncthreads();
  // the range's own first slots, for later
  const int own = s0 + lane < s1 ? idx[s0 + lane] : -1;
  const float own_w = s0 + lane < s1 ? wgt[s0 + lane] : 0.f;
#pragma unroll 4
  for (int i = threadIdx.x; i < slots; i += kGatherThreads) {
    const int e = idx[i];
    atomicAdd(&total[e], 1);
    if (i < s0) atomicAdd(&next[e], 1);
  }
  __syncthreads();
  if (warp == 0) {                                    // first row tile of every expert; next[e]: the row of the range's first slot for e
    int tiles = 0;
    for (int b = 0; b < E; b += 32) {
      const int e = b + lane, n = e < E ? total[e] : 0, mine = (n + 127) / 128;
      int upto = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += v;
      }
      const int t0 = tiles + upto - mine;
      if (e < E) {
        next[e] += t0 * 128;
        if (blockIdx.x == 0) {
          for (int i = 0; i < mine; ++i) tile_expert[t0 + i] = e;
          first[e] = t0 * 128;
        }
      }
      tiles += __shfl_sync(0xffffffffu, upto, 31);
    }
    if (blockIdx.x == 0 && lane == 0) *n_tiles = tiles;
  }
  if (blockIdx.x == 0) {                              // a warp per expert: the padding of its last tile
    __syncthreads();
    for (int e = warp; e < E; e += kGatherThreads / 32)
      for (int i = total[e] + lane; i < (total[e] + 127) / 128 * 128; i += 32) row_scale[first[e] + i] = 0.f;
  }
  for (int c0 = s0; c0 < s1; c0 += kGatherThreads) {
    const int c1 = min(c0 + kGatherThreads, s1);
    __syncthreads();
    if (warp == 0) {                                  // rows of the slots, in order
      for (int b = c0; b < c1; b += 32) {
        const int i = b + lane, e = b == s0 ? own : i < c1 ? idx[i] : -1;
        const uint32_t same = __match_any_sync(0xffffffffu, e);
        const int r = e >= 0 ? next[e] + __popc(same & ((1u << lane) - 1)) : 0;
        __syncwarp();
        if (e >= 0) {
          if (__ffs(same) == lane + 1) next[e] += __popc(same);
          row[i - c0] = r;
          pos[i] = r;
          row_scale[r] = b == s0 ? own_w : wgt[i];
        }
        __syncwarp();
      }
    }
    __syncthreads();
    for (int i = c0 + warp; i < c1; i += kGatherThreads / 32) {
      const uint4* src = h + (size_t)(i / top) * wv;
      uint4* dst = xs + (size_t)row[i - c0] * wv;
#pragma unroll 4
      for (int c = lane; c < wv; c += 32) dst[c] = src[c];
    }
  }
}

// acc[token] += sum over its slots of ys[pos[slot]]; a CTA per token, 8 columns a thread (W a multiple of 8).  Indexed through 64-bit
// divisions, four columns a thread, 3777 tokens of 2048 took 20 us where this takes 15.
__global__ void moe_combine_kernel(const __nv_bfloat16* __restrict__ ys, const int* __restrict__ pos, float* __restrict__ acc, int top,
                                   int W) {
  chain_enter(ys, pos, acc);
  const int* p = pos + (size_t)blockIdx.x * top;
  float* a = acc + (size_t)blockIdx.x * W;
  for (int c = threadIdx.x * 8; c < W; c += blockDim.x * 8) {
    float s[8];
    load_v<8>(a + c, s);
    for (int k = 0; k < top; ++k) {
      float f[8];
      load_v<8>(ys + (size_t)p[k] * W + c, f);
#pragma unroll
      for (int j = 0; j < 8; ++j) s[j] += f[j];
    }
    store_v<8>(a + c, s);
  }
}

}  // namespace ell

using namespace ell;

// out[b] (M x N, rows of ldo) = x[b] (M x K, rows of ldx) · w[b] (N x K contiguous)^T, `batch` products with the given
// element strides.  out_f32 / accumulate: fp32 output / added to an fp32 output; else the activation type.
ELL_API int ell_matvec(const void* x, const void* w, const void* bias, void* out, long long xb, long long wb, long long ob,
                       int batch, int M, int N, int K, int ldx, int ldo, int out_f32, int accumulate, int act_tanh,
                       int is_bf16, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || batch <= 0) return 0;
  if (batch > 65535) return -2;
  MatvecArgs a{x, w, bias, out, xb, wb, ob, M, N, K, ldx, ldo, out_f32, accumulate, act_tanh, 1};
  const int esz = is_bf16 ? 2 : 4;
  const bool vec = K % 8 == 0 && (ldx * esz) % 16 == 0 && aligned_to(x, 16) && aligned_to(w, 16) && (xb * esz) % 16 == 0 &&
                   (wb * esz) % 16 == 0;
  if (is_bf16 && vec) return launch_matvec_mma(a, batch, stream);
  return is_bf16 ? dispatch_matvec<__nv_bfloat16>(a, batch, vec, stream) : dispatch_matvec<float>(a, batch, vec, stream);
}

ELL_API int ell_moe_route(const float* z, const float* bias, int* idx, float* w, int n, int E, int top, int ldz, int softmax,
                          cudaStream_t stream) {
  if (n <= 0) return 0;
  if (E > 1024 || top > E || top < 1) return -2;
  launch_chained(moe_route_kernel, (n + 7) / 8, 256, 0, stream, z, bias, idx, w, n, E, top, ldz, softmax);
  return launch_status();
}

// z [n, N] = x w^T (rows of ldz), and the routing of its first E columns: bf16 x [n, K] (rows of ldx) and w [N, K], N up to 64, K a
// multiple of 8, 16-byte rows.
ELL_API int ell_moe_router(const void* x, const void* w, const float* bias, float* z, int* idx, float* score, int n, int N, int K,
                           int ldx, int ldz, int E, int top, int softmax, cudaStream_t stream) {
  if (n <= 0) return 0;
  if (N < 1 || N > 64 || E > N || top > E || top < 1 || top > 16 || K % 8 || ldx % 8 || !aligned_to(x, 16) || !aligned_to(w, 16)) return -2;
  auto kern = N <= 8 ? moe_router_kernel<1> : N <= 16 ? moe_router_kernel<2> : N <= 32 ? moe_router_kernel<4> : moe_router_kernel<8>;
  launch_chained(kern, (n + 15) / 16, kMvWarps * 32, 0, stream, (const __nv_bfloat16*)x, (const __nv_bfloat16*)w, bias, z, idx, score, n, N,
                 K, ldx, ldz, E, top, softmax);
  return launch_status();
}

// acc [n, W] fp32 += experts; up [E, F, W], down [E, W, F]; hid: scratch [n * top, F] of the activation type.
// glu_block > 0: gated experts, up [E, 2 F, W] with gate and up rows in alternating blocks of glu_block (a divisor of F).
ELL_API int ell_moe_rows(const void* h, const void* up, const void* down, const int* idx, const float* w, void* hid,
                         float* acc, int n, int top, int F, int W, int glu_block, int is_bf16, cudaStream_t stream) {
  if (n <= 0) return 0;
  if ((long long)n * top > 65535) return -2;
  const bool v = F % 8 == 0 && W % 8 == 0 && aligned_to(h, 16) && aligned_to(up, 16) && aligned_to(down, 16) && aligned_to(hid, 16);
  if (glu_block < 0 || (glu_block > 0 && F % glu_block)) return -2;
  dim3 gu(glu_block ? (F + 7) / 8 : (F + 15) / 16, n * top), gd((W + 15) / 16, n);
#define ELL_MOE_ROWS(T, V)                                                                                          \
  if (glu_block) launch_chained(moe_up_kernel<T, V, true>, gu, 256, 0, stream, (const T*)h, (const T*)up, idx, w, (T*)hid, top, F, W, glu_block); \
  else launch_chained(moe_up_kernel<T, V, false>, gu, 256, 0, stream, (const T*)h, (const T*)up, idx, w, (T*)hid, top, F, W, 1); \
  launch_chained(moe_down_kernel<T, V>, gd, 256, 0, stream, (const T*)hid, (const T*)down, idx, acc, top, F, W);
  if (is_bf16) {
    if (v) { ELL_MOE_ROWS(__nv_bfloat16, true) } else { ELL_MOE_ROWS(__nv_bfloat16, false) }
  } else {
    if (v) { ELL_MOE_ROWS(float, true) } else { ELL_MOE_ROWS(float, false) }
  }
#undef ELL_MOE_ROWS
  return launch_status();
}

// Row plan + gathered rows of the grouped GEMM (bf16, W a multiple of 8).
ELL_API int ell_moe_gather(const void* h, void* xs, const int* idx, const float* w, int* pos, float* row_scale,
                           int* tile_expert, int* n_tiles, int n, int top, int E, int W, cudaStream_t stream) {
  if (n <= 0) return 0;
  if (E > 1024 || W % 8) return -2;
  const int slots = n * top, grid = slots < 8 * kNumSMs ? (slots + 7) / 8 : 2 * kNumSMs;   // 8 slots a CTA until two CTAs fill an SM
  launch_chained(moe_gather_kernel, grid, kGatherThreads, 0, stream, (const uint4*)h, (uint4*)xs, idx, w, pos, row_scale, tile_expert,
                 n_tiles, slots, top, E, W / 8);
  return launch_status();
}

ELL_API int ell_moe_combine(const void* ys, const int* pos, float* acc, int n, int top, int W, cudaStream_t stream) {
  if (n <= 0) return 0;
  if (W % 8) return -2;
  launch_chained(moe_combine_kernel, n, W >= 2048 ? 256 : (W / 8 + 31) / 32 * 32, 0, stream, (const __nv_bfloat16*)ys, pos, acc, top, W);
  return launch_status();
}
