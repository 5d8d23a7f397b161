// A decoder layer of a training step, forward and backward, issued by one call each.
//
// Through modules and autograd functions a launch costs the host 25 us, so that a small batch waits for it: 200 tokens of 1024 in two
// layers ran their kernels in 550 us of 2450.  The kernels, their order and their routes are those of the single functions, with one
// sum less: where a layer's input is also its residual stream, both gradients meet in the norm's backward pass.
#include "vec.cuh"

ELL_API int ell_rmsnorm_fwd(const void* x, const void* res, const void* w, void* y, void* h_out, float* rstd, int rows, int cols,
                            float eps, cudaStream_t stream);
ELL_API int ell_rmsnorm_bwd(const void* dy, const void* h, const void* w, const float* rstd, const void* dres, void* dh, float* dw,
                            float* scratch, int rows, int cols, int accumulate_dw, cudaStream_t stream);
ELL_API int ell_rope(void* qkv, const float* cos_t, const float* sin_t, const int* pos, int T, int row_stride, int n_rot_heads, int D,
                     int backward, int table_rows, int* err, cudaStream_t stream);
ELL_API int ell_swiglu_fwd(const void* gu, void* out, int T, int F, cudaStream_t stream);
ELL_API int ell_swiglu_bwd(const void* dout, const void* gu, void* dgu, int T, int F, cudaStream_t stream);
ELL_API int ell_gemm_thin_route(int T, int N, int K);
ELL_API int ell_gemm_thin(const void* x, const void* W, void* out, const void* bias, int T, int N, int K, int ldx, int ldw, int ldo,
                          int w_mn, int out_mode, int split, int wait_us, int mute, int* err, cudaStream_t stream);
ELL_API int ell_gemm_bf16(const void* A, const void* B, void* C, const void* bias, int M, int N, int K, int lda, int ldb, int ldc,
                          int a_mn, int b_mn, int out_mode, int bn_hint, int* err, cudaStream_t stream);
ELL_API int ell_gemm_bf16_pair(const void* A, const void* B, void* C, const void* bias, int M, int N, int K, int lda, int ldb, int ldc,
                               int a_mn, int b_mn, int out_mode, int* err, cudaStream_t stream);
ELL_API int ell_gemm_pair_route(int M, int N);
ELL_API int ell_gemm_pair_refused(int rc);
ELL_API int ell_flash_attn_fwd(const void* q, const void* k, const void* v, void* out, float* lse, const int* row_start, int T, int Hq,
                               int Hk, int d, int dv, int q_stride, int k_stride, int v_stride, float scale, const float* alibi_slopes,
                               const float* sink, int window, int* err, cudaStream_t stream);
ELL_API int ell_flash_attn_bwd(const void* q, const void* k, const void* v, const void* out, const void* dout, const float* lse,
                               const int* row_start, void* dq, void* dk, void* dv, float* delta, float* dkv_acc, int T, int Hq, int Hk,
                               int q_stride, int kv_stride, int dq_stride, int dkv_stride, float scale, const float* alibi_slopes,
                               int* err, cudaStream_t stream);

namespace ell {

// The layer and what its forward pass leaves for the backward: everything but the two results lies in one buffer, `kept`.
struct TrainLayer {
  const void *qkv, *o, *gate_up, *down, *norm1, *norm2;                        // weights
  float *g_qkv, *g_o, *g_gate_up, *g_down, *g_norm1, *g_norm2;                 // their fp32 gradients, added to (backward); null: it ends in front of that step
  const void *x, *residual;       // [T, W]; residual null: x is the stream as well
  void *y, *h;                    // [T, W]: the layer's own result; the stream in front of the second norm
  void *kept;                     // ell_decoder_layer_kept bytes, on a 256-byte boundary
  const void *dy, *dh;            // gradients of y and h (backward)
  void *dx, *work;                // gradient of x and of the residual; ell_decoder_layer_work bytes (backward)
  float *norm_scratch, *delta, *kv_acc;
  const float *cos, *sin, *slopes;        // tables and slopes, or null
  const int *pos, *row_start;
  int* err;
  long long T, W, Hq, Hk, F, table_rows;
  long long pairs;                // whether products may run on CTA pairs; 0 after a launch that was refused
  long long launches, failed;
};
static_assert(sizeof(TrainLayer) == 39 * 8, "the caller lays it out as 64-bit words");
constexpr int kTrD = 128;                            // head size
enum TrainPart { kTrNorm = 1, kTrProduct, kTrRotation, kTrAttention, kTrActivation };

static int tr_product(TrainLayer& a, const void* x, const void* w, void* out, long long M_, long long N_, long long K_, int lda, int ldb,
                      int a_mn, int b_mn, int out_mode, cudaStream_t stream) {
  const int M = (int)M_, N = (int)N_, K = (int)K_;
  if (a.pairs && ell_gemm_pair_route(M, N)) {
    const int rc = ell_gemm_bf16_pair(x, w, out, nullptr, M, N, K, lda, ldb, N, a_mn, b_mn, out_mode, a.err, stream);
    if (!ell_gemm_pair_refused(rc)) return rc;
    a.pairs = 0;                                       // nothing was launched: on single CTAs from here on
  }
  return ell_gemm_bf16(x, w, out, nullptr, M, N, K, lda, ldb, N, a_mn, b_mn, out_mode, 0, a.err, stream);
}
// out [T, N] = x [T, K] w [N, K]^T; dx [T, K] = dy [T, N] w; dw [N, K] += dy^T x
static int tr_forward(TrainLayer& a, const void* x, const void* w, void* out, long long N, long long K, cudaStream_t stream) {
  return tr_product(a, x, w, out, a.T, N, K, (int)K, (int)K, 0, 0, 0, stream);
}
static int tr_input(TrainLayer& a, const void* dy, const void* w, void* dx, long long N, long long K, cudaStream_t stream) {
  if (ell_gemm_thin_route((int)a.T, (int)K, (int)N))
    return ell_gemm_thin(dy, w, dx, nullptr, (int)a.T, (int)K, (int)N, (int)N, (int)K, (int)K, 1, 0, 0, 0, -1, a.err, stream);
  return tr_product(a, dy, w, dx, a.T, K, N, (int)N, (int)K, 0, 1, 0, stream);
}
static int tr_weight(TrainLayer& a, const void* dy, const void* x, float* dw, long long N, long long K, cudaStream_t stream) {
  return tr_product(a, dy, x, dw, N, K, a.T, (int)N, (int)K, 1, 1, 1, stream);
}

struct TrainKept {
  size_t h1, rstd1, n1, qkv, att, lse, rstd2, n2, gate_up, act, bytes;
};
struct TrainWork {
  size_t wide, dn, dh2, datt, dqkv, bytes;
};
struct Places {
  size_t at = 0;
  size_t take(size_t bytes) {
    const size_t p = at;
    at += (bytes + 255) / 256 * 256;
    return p;
  }
};
static TrainKept tr_kept(const TrainLayer& a) {
  TrainKept k{};
  Places p;
  const size_t T = a.T, row = T * a.W * 2;
  if (a.residual) k.h1 = p.take(row);
  k.rstd1 = p.take(T * 4);
  k.n1 = p.take(row);
  k.qkv = p.take(T * (a.Hq + 2 * a.Hk) * kTrD * 2);
  k.att = p.take(T * a.Hq * kTrD * 2);
  k.lse = p.take(T * a.Hq * 4);
  k.rstd2 = p.take(T * 4);
  k.n2 = p.take(row);
  k.gate_up = p.take(T * 2 * a.F * 2);
  k.act = p.take(T * a.F * 2);
  k.bytes = p.at;
  return k;
}
// The gradients of the activation and of its input, then those of the attention.
static TrainWork tr_work(const TrainLayer& a) {
  TrainWork w{};
  Places p;
  const size_t T = a.T, row = T * a.W * 2;
  w.dn = p.take(row);
  w.dh2 = p.take(row);
  const size_t shared = p.at;
  w.datt = p.take(T * a.Hq * kTrD * 2);
  w.dqkv = p.take(T * (a.Hq + 2 * a.Hk) * kTrD * 2);
  const size_t end = p.at;
  p.at = shared;
  w.wide = p.take(T * a.F * 2);
  p.take(T * 2 * a.F * 2);
  w.bytes = p.at > end ? p.at : end;
  return w;
}

#define ELL_TR(part_, n, call)                             \
  if ((rc = (call)) != 0) return a.failed = part_, rc;     \
  a.launches += n

static int train_forward(TrainLayer& a, float eps, float scale, cudaStream_t s) {
  const TrainKept at = tr_kept(a);
  char* k = static_cast<char*>(a.kept);
  const int T = (int)a.T, W = (int)a.W, Hq = (int)a.Hq, Hk = (int)a.Hk, F = (int)a.F, D = kTrD, ld = (Hq + 2 * Hk) * D;
  __nv_bfloat16* qkv = reinterpret_cast<__nv_bfloat16*>(k + at.qkv);
  const void* h1 = a.residual ? k + at.h1 : a.x;
  int rc;
  ELL_TR(kTrNorm, 1, ell_rmsnorm_fwd(a.x, a.residual, a.norm1, k + at.n1, a.residual ? k + at.h1 : nullptr, (float*)(k + at.rstd1), T, W, eps, s));
  ELL_TR(kTrProduct, 1, tr_forward(a, k + at.n1, a.qkv, qkv, ld, W, s));
  if (a.cos) {
    ELL_TR(kTrRotation, 1, ell_rope(qkv, a.cos, a.sin, a.pos, T, ld, Hq + Hk, D, 0, (int)a.table_rows, a.err, s));
  }
  ELL_TR(kTrAttention, 1, ell_flash_attn_fwd(qkv, qkv + Hq * D, qkv + (Hq + Hk) * D, k + at.att, (float*)(k + at.lse), a.row_start, T, Hq, Hk,
                                             D, D, ld, ld, ld, scale, a.slopes, nullptr, 0, a.err, s));
  ELL_TR(kTrProduct, 1, tr_forward(a, k + at.att, a.o, a.y, W, Hq * D, s));
  ELL_TR(kTrNorm, 1, ell_rmsnorm_fwd(a.y, h1, a.norm2, k + at.n2, a.h, (float*)(k + at.rstd2), T, W, eps, s));
  ELL_TR(kTrProduct, 1, tr_forward(a, k + at.n2, a.gate_up, k + at.gate_up, 2 * F, W, s));
  ELL_TR(kTrActivation, 1, ell_swiglu_fwd(k + at.gate_up, k + at.act, T, F, s));
  ELL_TR(kTrProduct, 1, tr_forward(a, k + at.act, a.down, a.y, W, F, s));
  return 0;
}

static int train_backward(TrainLayer& a, float scale, cudaStream_t s) {
  const TrainKept at = tr_kept(a);
  const TrainWork to = tr_work(a);
  char *k = static_cast<char*>(a.kept), *w = static_cast<char*>(a.work);
  const int T = (int)a.T, W = (int)a.W, Hq = (int)a.Hq, Hk = (int)a.Hk, F = (int)a.F, D = kTrD, ld = (Hq + 2 * Hk) * D;
  const __nv_bfloat16* qkv = reinterpret_cast<const __nv_bfloat16*>(k + at.qkv);
  __nv_bfloat16* dqkv = reinterpret_cast<__nv_bfloat16*>(w + to.dqkv);
  void *dact = w + to.wide, *dgu = w + to.wide + ((size_t)T * F * 2 + 255) / 256 * 256, *dn = w + to.dn, *dh2 = w + to.dh2, *datt = w + to.datt;
  const void* h1 = a.residual ? k + at.h1 : a.x;
  int rc;
  ELL_TR(kTrProduct, 1, tr_input(a, a.dy, a.down, dact, W, F, s));
  ELL_TR(kTrProduct, 1, tr_weight(a, a.dy, k + at.act, a.g_down, W, F, s));
  if (!a.g_gate_up) return 0;
  ELL_TR(kTrActivation, 1, ell_swiglu_bwd(dact, k + at.gate_up, dgu, T, F, s));
  ELL_TR(kTrProduct, 1, tr_input(a, dgu, a.gate_up, dn, 2 * F, W, s));
  ELL_TR(kTrProduct, 1, tr_weight(a, dgu, k + at.n2, a.g_gate_up, 2 * F, W, s));
  if (!a.g_norm2) return 0;
  ELL_TR(kTrNorm, 2, ell_rmsnorm_bwd(dn, a.h, a.norm2, (const float*)(k + at.rstd2), a.dh, dh2, a.g_norm2, a.norm_scratch, T, W, 1, s));
  if (!a.g_o) return 0;
  ELL_TR(kTrProduct, 1, tr_input(a, dh2, a.o, datt, W, Hq * D, s));
  ELL_TR(kTrProduct, 1, tr_weight(a, dh2, k + at.att, a.g_o, W, Hq * D, s));
  if (!a.g_qkv) return 0;
  ELL_TR(kTrAttention, 3, ell_flash_attn_bwd(qkv, qkv + Hq * D, qkv + (Hq + Hk) * D, k + at.att, datt, (const float*)(k + at.lse), a.row_start,
                                             dqkv, dqkv + Hq * D, dqkv + (Hq + Hk) * D, a.delta, a.kv_acc, T, Hq, Hk, ld, ld, ld, ld, scale,
                                             a.slopes, a.err, s));
  if (a.cos) {
    ELL_TR(kTrRotation, 1, ell_rope(dqkv, a.cos, a.sin, a.pos, T, ld, Hq + Hk, D, 1, (int)a.table_rows, a.err, s));
  }
  ELL_TR(kTrProduct, 1, tr_input(a, dqkv, a.qkv, dn, ld, W, s));
  ELL_TR(kTrProduct, 1, tr_weight(a, dqkv, k + at.n1, a.g_qkv, ld, W, s));
  if (!a.g_norm1) return 0;
  ELL_TR(kTrNorm, 2, ell_rmsnorm_bwd(dn, h1, a.norm1, (const float*)(k + at.rstd1), dh2, a.dx, a.g_norm1, a.norm_scratch, T, W, 1, s));
  return 0;
}
#undef ELL_TR

}  // namespace ell

using namespace ell;

ELL_API long long ell_decoder_layer_kept(const long long* args) { return (long long)tr_kept(*reinterpret_cast<const TrainLayer*>(args)).bytes; }
ELL_API long long ell_decoder_layer_work(const long long* args) { return (long long)tr_work(*reinterpret_cast<const TrainLayer*>(args)).bytes; }

// args: the words of TrainLayer; heads of 128; W and F multiples of 8, all on 16-byte boundaries.  backward 0: y, h and `kept` from x and
// residual; 1: dx, and the weights' gradients added to, from dy and dh.
ELL_API int ell_decoder_layer(long long* args, int backward, float eps, float scale, cudaStream_t stream) {
  TrainLayer& a = *reinterpret_cast<TrainLayer*>(args);
  a.launches = a.failed = 0;
  if (a.T <= 0) return 0;
  if (a.W % 8 || a.F % 8 || !aligned_to(a.kept, 256) || (backward && !aligned_to(a.work, 256))) return -2;
  return backward ? train_backward(a, scale, stream) : train_forward(a, eps, scale, stream);
}
