// RoPE and SwiGLU kernels for sm_100a (HBM-bound elementwise ops, 16-byte vector access).
//
// RoPE is applied in place on the q and k heads of the packed QKV GEMM output
// `[T, (Hq + 2·Hk) · D]` (NeoX half rotation, positions gathered per token so packed documents
// restart at 0).  The backward is the same rotation with -sin.  Replaces the eager /
// Triton rotary of the reference (llm/models/mg_models/llama/positional_embeddings.py:94-122).
//
// SwiGLU reads the fused gate|up GEMM output `[T, 2F]` (gate columns first) and writes
// `silu(gate) * up` `[T, F]`; the backward recomputes the activation from gate|up
// (llm/models/mg_models/llama/transformer.py:217-225 materialises both halves and the SiLU).
#include "common.cuh"

namespace ell {

// One thread rotates 8 (x1) + 8 (x2) elements of one head: D/2 must be a multiple of 8.
// A position outside the cos / sin tables is reported through the error word (code 32) and its row left unrotated,
// instead of reading past the tables.
__global__ void rope_kernel(__nv_bfloat16* __restrict__ qkv, const float* __restrict__ cos_t,
                            const float* __restrict__ sin_t, const int* __restrict__ pos, int T, int row_stride,
                            int n_rot_heads, int D, float sin_sign, int table_rows, int* __restrict__ err) {
  chain_enter(qkv, cos_t, sin_t, pos, err);
  const int half = D / 2, vec_per_head = half / 8;
  const long long total = (long long)T * n_rot_heads * vec_per_head;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int v = (int)(i % vec_per_head);
    const int hd = (int)((i / vec_per_head) % n_rot_heads);
    const int t = (int)(i / ((long long)vec_per_head * n_rot_heads));
    const int p = pos[t];
    if (p < 0 || p >= table_rows) {
      if (err != nullptr) atomicCAS(err, 0, 32);
      continue;
    }
    __nv_bfloat16* base = qkv + (size_t)t * row_stride + (size_t)hd * D + v * 8;
    float x1[8], x2[8], c[8], s[8];
    unpack8(*reinterpret_cast<const bf16x8*>(base), x1);
    unpack8(*reinterpret_cast<const bf16x8*>(base + half), x2);
    const float4* cp = reinterpret_cast<const float4*>(cos_t + (size_t)p * half + v * 8);
    const float4* sp = reinterpret_cast<const float4*>(sin_t + (size_t)p * half + v * 8);
    float4 c0 = cp[0], c1 = cp[1], s0 = sp[0], s1 = sp[1];
    c[0] = c0.x; c[1] = c0.y; c[2] = c0.z; c[3] = c0.w; c[4] = c1.x; c[5] = c1.y; c[6] = c1.z; c[7] = c1.w;
    s[0] = s0.x; s[1] = s0.y; s[2] = s0.z; s[3] = s0.w; s[4] = s1.x; s[5] = s1.y; s[6] = s1.z; s[7] = s1.w;
    float o1[8], o2[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float sj = s[j] * sin_sign;
      o1[j] = x1[j] * c[j] - x2[j] * sj;
      o2[j] = x2[j] * c[j] + x1[j] * sj;
    }
    *reinterpret_cast<bf16x8*>(base) = pack8(o1);
    *reinterpret_cast<bf16x8*>(base + half) = pack8(o2);
  }
}

// rope_kernel on the q and k heads of rows [q | k | v], with the rotated keys and the values also written to their places in a
// cache: token t's to row base[t] + len[t] - 1.  A step of a few rows is bound by its launches (decoding: 2.3 us here and 1.4 for
// the copy) and by the host's calls (a short prompt), a prompt by the keys and values that were read twice: 4096 rows of 32 + 2 x 8
// heads took 22.9 + 11.3 us.
__global__ void rope_append_kernel(__nv_bfloat16* __restrict__ qkv, const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                                   const int* __restrict__ pos, __nv_bfloat16* __restrict__ kc, __nv_bfloat16* __restrict__ vc,
                                   const int* __restrict__ base, const int* __restrict__ len, int T, int Hq, int Hk, int D,
                                   int table_rows, int* __restrict__ err) {
  chain_enter(qkv, cos_t, sin_t, pos, kc, vc, base, len, err);
  const int half = D / 2, rot = (Hq + Hk) * (half / 8), per = rot + Hk * (D / 8), W = (Hq + 2 * Hk) * D;
  const long long total = (long long)T * per;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int t = (int)(i / per), c = (int)(i % per);
    __nv_bfloat16* row = qkv + (size_t)t * W;
    const size_t place = ((size_t)base[t] + len[t] - 1) * Hk * D;
    if (c >= rot) {
      const int at = (c - rot) * 8;
      *reinterpret_cast<bf16x8*>(vc + place + at) = *reinterpret_cast<const bf16x8*>(row + (size_t)(Hq + Hk) * D + at);
      continue;
    }
    const int hd = c / (half / 8), v = c % (half / 8) * 8, p = pos[t];
    __nv_bfloat16* x = row + (size_t)hd * D + v;
    bf16x8 lo = *reinterpret_cast<const bf16x8*>(x), hi = *reinterpret_cast<const bf16x8*>(x + half);
    if (p < 0 || p >= table_rows) {
      if (err != nullptr) atomicCAS(err, 0, 32);
    } else {
      float x1[8], x2[8], o1[8], o2[8];
      unpack8(lo, x1);
      unpack8(hi, x2);
#pragma unroll
      for (int j = 0; j < 8; j += 4) {
        const float4 cs = *reinterpret_cast<const float4*>(cos_t + (size_t)p * half + v + j);
        const float4 sn = *reinterpret_cast<const float4*>(sin_t + (size_t)p * half + v + j);
        const float cj[4] = {cs.x, cs.y, cs.z, cs.w}, sj[4] = {sn.x, sn.y, sn.z, sn.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          o1[j + e] = x1[j + e] * cj[e] - x2[j + e] * sj[e];
          o2[j + e] = x2[j + e] * cj[e] + x1[j + e] * sj[e];
        }
      }
      lo = pack8(o1);
      hi = pack8(o2);
      *reinterpret_cast<bf16x8*>(x) = lo;
      *reinterpret_cast<bf16x8*>(x + half) = hi;
    }
    if (hd >= Hq) {
      __nv_bfloat16* k = kc + place + (size_t)(hd - Hq) * D + v;
      *reinterpret_cast<bf16x8*>(k) = lo;
      *reinterpret_cast<bf16x8*>(k + half) = hi;
    }
  }
}

__global__ void swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ out, int T, int F) {
  chain_enter(gu, out);
  const int fv = F / 8;
  const long long total = (long long)T * fv;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int t = (int)(i / fv), c = (int)(i % fv);
    float g[8], u[8], o[8];
    unpack8(reinterpret_cast<const bf16x8*>(gu + (size_t)t * 2 * F)[c], g);
    unpack8(reinterpret_cast<const bf16x8*>(gu + (size_t)t * 2 * F + F)[c], u);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = g[j] / (1.f + __expf(-g[j])) * u[j];
    reinterpret_cast<bf16x8*>(out + (size_t)t * F)[c] = pack8(o);
  }
}

__global__ void swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ gu,
                                  __nv_bfloat16* __restrict__ dgu, int T, int F) {
  const int fv = F / 8;
  const long long total = (long long)T * fv;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int t = (int)(i / fv), c = (int)(i % fv);
    float g[8], u[8], d[8], dg[8], du[8];
    unpack8(reinterpret_cast<const bf16x8*>(gu + (size_t)t * 2 * F)[c], g);
    unpack8(reinterpret_cast<const bf16x8*>(gu + (size_t)t * 2 * F + F)[c], u);
    unpack8(reinterpret_cast<const bf16x8*>(dout + (size_t)t * F)[c], d);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float sg = 1.f / (1.f + __expf(-g[j]));
      const float silu = g[j] * sg;
      du[j] = d[j] * silu;
      dg[j] = d[j] * u[j] * sg * (1.f + g[j] * (1.f - sg));
    }
    reinterpret_cast<bf16x8*>(dgu + (size_t)t * 2 * F)[c] = pack8(dg);
    reinterpret_cast<bf16x8*>(dgu + (size_t)t * 2 * F + F)[c] = pack8(du);
  }
}

// out(fp32) += in(bf16): gradient accumulation of one parameter into the fp32 flat buffer.
__global__ void accum_bf16_to_f32_kernel(const __nv_bfloat16* __restrict__ in, float* __restrict__ out, long long n) {
  const long long nv = n / 8;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nv;
       i += (long long)gridDim.x * blockDim.x) {
    float f[8];
    unpack8(reinterpret_cast<const bf16x8*>(in)[i], f);
    float4* o = reinterpret_cast<float4*>(out) + 2 * i;
    float4 a = o[0], b = o[1];
    a.x += f[0]; a.y += f[1]; a.z += f[2]; a.w += f[3];
    b.x += f[4]; b.y += f[5]; b.z += f[6]; b.w += f[7];
    o[0] = a; o[1] = b;
  }
  if (blockIdx.x == 0 && threadIdx.x < (n & 7)) {
    const long long j = nv * 8 + threadIdx.x;
    out[j] += __bfloat162float(in[j]);
  }
}

inline int ew_grid(long long work_items, int threads) {
  long long b = (work_items + threads - 1) / threads;
  long long cap = (long long)kNumSMs * 16;
  return (int)(b < 1 ? 1 : (b < cap ? b : cap));
}

}  // namespace ell

using namespace ell;

// cos_t / sin_t: fp32 [table_rows, D/2]; positions outside [0, table_rows) set *err to 32.
ELL_API int ell_rope(void* qkv, const float* cos_t, const float* sin_t, const int* pos, int T, int row_stride,
                     int n_rot_heads, int D, int backward, int table_rows, int* err, cudaStream_t stream) {
  if (D % 16) return -1;
  long long total = (long long)T * n_rot_heads * (D / 16);
  if (total == 0) return 0;
  launch_chained(rope_kernel, ew_grid(total, 256), 256, 0, stream, (__nv_bfloat16*)qkv, cos_t, sin_t, pos, T, row_stride,
                                                       n_rot_heads, D, backward ? -1.f : 1.f, table_rows, err);
  return launch_status();
}

// qkv: contiguous rows of (Hq + 2 Hk) heads of D; kc, vc: rows of Hk D.
ELL_API int ell_rope_append(void* qkv, const float* cos_t, const float* sin_t, const int* pos, void* kc, void* vc, const int* base,
                            const int* len, int T, int Hq, int Hk, int D, int table_rows, int* err, cudaStream_t stream) {
  if (D % 16) return -1;
  const long long total = (long long)T * ((Hq + Hk) * (D / 16) + Hk * (D / 8));
  if (total == 0) return 0;
  launch_chained(rope_append_kernel, ew_grid(total, 256), 256, 0, stream, (__nv_bfloat16*)qkv, cos_t, sin_t, pos, (__nv_bfloat16*)kc,
                 (__nv_bfloat16*)vc, base, len, T, Hq, Hk, D, table_rows, err);
  return launch_status();
}

ELL_API int ell_swiglu_fwd(const void* gu, void* out, int T, int F, cudaStream_t stream) {
  if (F % 8) return -1;
  long long total = (long long)T * (F / 8);
  if (total == 0) return 0;
  launch_chained(swiglu_fwd_kernel, ew_grid(total, 256), 256, 0, stream, (const __nv_bfloat16*)gu, (__nv_bfloat16*)out, T, F);
  return launch_status();
}

ELL_API int ell_swiglu_bwd(const void* dout, const void* gu, void* dgu, int T, int F, cudaStream_t stream) {
  if (F % 8) return -1;
  long long total = (long long)T * (F / 8);
  if (total == 0) return 0;
  swiglu_bwd_kernel<<<ew_grid(total, 256), 256, 0, stream>>>((const __nv_bfloat16*)dout, (const __nv_bfloat16*)gu,
                                                            (__nv_bfloat16*)dgu, T, F);
  return launch_status();
}

ELL_API int ell_accum_bf16_to_f32(const void* in, float* out, long long n, cudaStream_t stream) {
  if (n == 0) return 0;
  accum_bf16_to_f32_kernel<<<ew_grid(n / 8 + 1, 256), 256, 0, stream>>>((const __nv_bfloat16*)in, out, n);
  return launch_status();
}

// ---------------------------------------------------------------------------------------------
// Vocab-parallel embedding: masked row gather, and its backward as an fp32 scatter-add straight
// into the weight's gradient accumulator (no bf16 gradient tensor, no sort).
// Replaces F.embedding + mask writes of the reference
// (llm/models/mg_models/base_modules/layers/vocab_parallel_emb.py:106-137).
// ---------------------------------------------------------------------------------------------
namespace ell {

// out[t, :] = ids[t] in [vocab_start, vocab_start + rows) ? weight[ids[t] - vocab_start, :] : 0
// An id outside [0, vocab_total) is reported through the error word (code 31) instead of a host-side max() of the
// ids, which would cost a device synchronisation per micro-batch; its row is written as zeros.
__global__ void embedding_fwd_kernel(const long long* __restrict__ ids, const __nv_bfloat16* __restrict__ weight,
                                     __nv_bfloat16* __restrict__ out, int T, int cols, long long vocab_start,
                                     long long rows, long long vocab_total, int* __restrict__ err) {
  const int nvec = cols / 8;
  for (int t = blockIdx.x; t < T; t += gridDim.x) {
    const long long id = ids[t];
    if (err != nullptr && threadIdx.x == 0 && (id < 0 || id >= vocab_total)) atomicCAS(err, 0, 31);
    const long long loc = id - vocab_start;
    const bool mine = loc >= 0 && loc < rows;
    const bf16x8* src = reinterpret_cast<const bf16x8*>(weight + (mine ? loc : 0) * cols);
    bf16x8* dst = reinterpret_cast<bf16x8*>(out + (size_t)t * cols);
    for (int c = threadIdx.x; c < nvec; c += blockDim.x) dst[c] = mine ? src[c] : bf16x8{};
  }
}

// grad32[ids[t] - vocab_start, :] += dout[t, :] for the ids this rank owns (fp32 vector atomics)
__global__ void embedding_bwd_kernel(const long long* __restrict__ ids, const __nv_bfloat16* __restrict__ dout,
                                     float* __restrict__ grad32, int T, int cols, long long vocab_start,
                                     long long rows) {
  const int nvec = cols / 8;
  for (int t = blockIdx.x; t < T; t += gridDim.x) {
    const long long loc = ids[t] - vocab_start;
    if (loc < 0 || loc >= rows) continue;
    const bf16x8* src = reinterpret_cast<const bf16x8*>(dout + (size_t)t * cols);
    float* dst = grad32 + loc * cols;
    for (int c = threadIdx.x; c < nvec; c += blockDim.x) {
      float f[8];
      unpack8(src[c], f);
      atomicAdd(reinterpret_cast<float4*>(dst + c * 8), make_float4(f[0], f[1], f[2], f[3]));
      atomicAdd(reinterpret_cast<float4*>(dst + c * 8 + 4), make_float4(f[4], f[5], f[6], f[7]));
    }
  }
}

// The same with a fixed order of the sums.  Tokens come in blocks of kIdBlock; seen[id] has a bit for every block that holds the id.
// Up to kUnmarkedIds tokens are looked through whole instead: a small batch is bound by the host, and marking is two launches more.
constexpr int kIdBlock = 128, kIdWarps = kIdBlock / 32, kUnmarkedIds = 1024;
__global__ void embedding_mark_kernel(const long long* __restrict__ ids, uint32_t* __restrict__ seen, int T, int words, long long rows) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= T || ids[t] < 0 || ids[t] >= rows) return;
  atomicOr(seen + ids[t] * words + t / kIdBlock / 32, 1u << (t / kIdBlock & 31));
}

// The CTA at an id's first token adds up the id's rows in the order of the tokens, and adds the sum to the table's row, which no other
// CTA writes.  Four blocks that hold the id are looked through at a time, one a warp; a thread owns eight columns and has kRowsAhead
// rows in flight.  3001 tokens of 2048 40 us, 4096 of 4096 75 to 100.  (Atomics 12 and 28, but in no fixed order; a stable sort and its
// temporaries alone 45.)
constexpr int kRowsAhead = 16;
__global__ void __launch_bounds__(kIdBlock) embedding_bwd_ordered_kernel(const long long* __restrict__ ids, const uint32_t* __restrict__ seen,
                                                                         const __nv_bfloat16* __restrict__ dout,
                                                                         float* __restrict__ grad32, int T, int words, int cols,
                                                                         long long rows) {
  __shared__ int list[kIdWarps * kIdBlock], count[kIdWarps];
  const int t = blockIdx.x, own = t / kIdBlock, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long id = ids[t];
  if (id < 0 || id >= rows) return;
  const uint32_t* blocks = seen != nullptr ? seen + id * words : nullptr;
  int word = own / 32;
  uint32_t left;                                       // blocks still to look through
  bool earlier = false;
  if (blocks != nullptr) {
    left = blocks[word];
    for (int w = 0; w < word; ++w)
      if (blocks[w] != 0) return;
    if (left & ((1u << (own & 31)) - 1)) return;
    const int at = own * kIdBlock + threadIdx.x;
    earlier = at < t && ids[at] == id;
  } else {
    left = (1u << (T + kIdBlock - 1) / kIdBlock) - (1u << own);
    for (int i = threadIdx.x; i < t; i += kIdBlock) earlier |= ids[i] == id;
  }
  if (__syncthreads_or(earlier)) return;
  const int c = (blockIdx.y * kIdBlock + threadIdx.x) * 8;
  const __nv_bfloat16* src = dout + c;
  float acc[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) acc[e] = 0.f;
  while (true) {
    int mine = -1;                                     // this warp's block of the next four
    for (int n = 0; n < kIdWarps; ++n) {
      while (left == 0 && word + 1 < words) left = blocks[++word];
      if (left == 0) break;
      if (n == warp) mine = word * 32 + __ffs(left) - 1;
      left &= left - 1;
    }
    uint32_t same[kIdBlock / 32];
    int mine_count = 0;
#pragma unroll
    for (int q = 0; q < kIdBlock / 32; ++q) {
      const int tok = mine * kIdBlock + q * 32 + lane;
      same[q] = __ballot_sync(0xffffffffu, mine >= 0 && tok < T && ids[mine >= 0 && tok < T ? tok : 0] == id);
      mine_count += __popc(same[q]);
    }
    if (lane == 0) count[warp] = mine_count;
    __syncthreads();
    int total = 0, place = 0;
#pragma unroll
    for (int w = 0; w < kIdWarps; ++w) {
      if (w < warp) place += count[w];
      total += count[w];
    }
#pragma unroll
    for (int q = 0; q < kIdBlock / 32; ++q) {
      if (same[q] >> lane & 1) list[place + __popc(same[q] & ((1u << lane) - 1))] = mine * kIdBlock + q * 32 + lane;
      place += __popc(same[q]);
    }
    __syncthreads();
    if (total == 0) break;
    if (c < cols) {
      for (int i = 0; i < total; i += kRowsAhead) {
        bf16x8 x[kRowsAhead];
#pragma unroll
        for (int j = 0; j < kRowsAhead; ++j)
          if (i + j < total) x[j] = *reinterpret_cast<const bf16x8*>(src + (size_t)list[i + j] * cols);
#pragma unroll
        for (int j = 0; j < kRowsAhead; ++j) {
          if (i + j < total) {
            float f[8];
            unpack8(x[j], f);
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[e] += f[e];
          }
        }
      }
    }
    __syncthreads();                                   // before the next four are listed
  }
  if (c >= cols) return;
  float4* dst = reinterpret_cast<float4*>(grad32 + id * cols + c);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const float4 g = dst[h];
    dst[h] = make_float4(g.x + acc[4 * h], g.y + acc[4 * h + 1], g.z + acc[4 * h + 2], g.w + acc[4 * h + 3]);
  }
}

}  // namespace ell

// vocab_total > 0 with err != nullptr: ids outside [0, vocab_total) set *err to 31.
ELL_API int ell_embedding_fwd(const long long* ids, const void* weight, void* out, int T, int cols,
                              long long vocab_start, long long rows, long long vocab_total, int* err,
                              cudaStream_t stream) {
  if (T == 0) return 0;
  if (cols % 8) return -1;
  const int grid = T < ell::kNumSMs * 16 ? T : ell::kNumSMs * 16;
  ell::embedding_fwd_kernel<<<grid, 128, 0, stream>>>(ids, (const __nv_bfloat16*)weight, (__nv_bfloat16*)out, T, cols,
                                                       vocab_start, rows, vocab_total, vocab_total > 0 ? err : nullptr);
  return ell::launch_status();
}

ELL_API int ell_embedding_bwd(const long long* ids, const void* dout, float* grad32, int T, int cols,
                              long long vocab_start, long long rows, cudaStream_t stream) {
  if (T == 0) return 0;
  if (cols % 8) return -1;
  const int grid = T < ell::kNumSMs * 16 ? T : ell::kNumSMs * 16;
  ell::embedding_bwd_kernel<<<grid, 128, 0, stream>>>(ids, (const __nv_bfloat16*)dout, grad32, T, cols, vocab_start,
                                                       rows);
  return ell::launch_status();
}

// 32-bit words of work space a table row takes (0: none is needed).
ELL_API int ell_embedding_bwd_words(int T) {
  return T <= ell::kUnmarkedIds ? 0 : (T + 32 * ell::kIdBlock - 1) / (32 * ell::kIdBlock);
}

// seen: rows * ell_embedding_bwd_words(T) words of work space.
ELL_API int ell_embedding_bwd_ordered(const long long* ids, void* seen, const void* dout, float* grad32, int T, int cols, long long rows,
                                      cudaStream_t stream) {
  if (T <= 0) return 0;
  if (cols % 8) return -1;
  const int per = 8 * ell::kIdBlock, words = ell_embedding_bwd_words(T);
  if (cols > 65535 * per) return -2;
  if (words > 0) {
    const cudaError_t e = cudaMemsetAsync(seen, 0, (size_t)rows * words * 4, stream);
    if (e != cudaSuccess) return (int)e;
    ell::embedding_mark_kernel<<<(T + 255) / 256, 256, 0, stream>>>(ids, (uint32_t*)seen, T, words, rows);
  }
  ell::embedding_bwd_ordered_kernel<<<dim3(T, (cols + per - 1) / per), ell::kIdBlock, 0, stream>>>(
      ids, words > 0 ? (const uint32_t*)seen : nullptr, (const __nv_bfloat16*)dout, grad32, T, words, cols, rows);
  return ell::launch_status();
}

namespace ell {
// Column sums of a bf16 matrix added into fp32: out[c] += sum_r x[r, c].  The bias gradient of a linear layer
// (db = sum over tokens of dy) without materialising an fp32 copy of dy.  A block covers 256 columns (32 threads x 8
// columns, 16-byte loads) and a slice of the rows (8 row lanes); lanes meet in shared memory, one atomic per column
// and block.
__global__ void __launch_bounds__(256) colsum_kernel(const __nv_bfloat16* __restrict__ x, float* __restrict__ out,
                                                     int rows, int cols) {
  __shared__ float red[8][256];
  const int cg = threadIdx.x & 31, rl = threadIdx.x >> 5;
  const int c0 = blockIdx.x * 256 + cg * 8;
  float acc[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) acc[e] = 0.f;
  if (c0 < cols) {
    for (int r = blockIdx.y * 8 + rl; r < rows; r += gridDim.y * 8) {
      float t[8];
      unpack8(*reinterpret_cast<const bf16x8*>(x + (size_t)r * cols + c0), t);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] += t[e];
    }
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) red[rl][cg * 8 + e] = acc[e];
  __syncthreads();
  const int c = blockIdx.x * 256 + threadIdx.x;
  if (c < cols) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) s += red[i][threadIdx.x];
    atomicAdd(out + c, s);
  }
}
}  // namespace ell

// out[cols] (fp32) += column sums of x[rows, cols] (bf16, cols a multiple of 8).
ELL_API int ell_colsum_bf16(const void* x, float* out, int rows, int cols, cudaStream_t stream) {
  if (rows <= 0 || cols <= 0) return 0;
  if (cols % 8) return -1;
  const int bx = (cols + 255) / 256;
  int by = (rows + 63) / 64;
  const int cap = (ell::kNumSMs * 8 + bx - 1) / bx;
  if (by > cap) by = cap;
  if (by < 1) by = 1;
  ell::colsum_kernel<<<dim3(bx, by), 256, 0, stream>>>((const __nv_bfloat16*)x, out, rows, cols);
  return ell::launch_status();
}
