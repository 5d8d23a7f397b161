// The layers of a decoder in a serving step, issued by one call.
//
// From Python a launch costs 15 to 30 us of host time (modules, tensors, arguments through ctypes), which a short prompt waits for: 77
// tokens of 2048 through 4 layers ran their kernels in 350 us of 1250.  Here a launch costs what the driver takes, about 4 us.  The
// kernels, their order and their routes are those of the layers' own forward methods; only who calls them differs.
#include <algorithm>

#include "vec.cuh"

ELL_API int ell_rmsnorm_fwd(const void* x, const void* res, const void* w, void* y, void* h_out, float* rstd, int rows, int cols,
                            float eps, cudaStream_t stream);
ELL_API int ell_rope_append(void* qkv, const float* cos_t, const float* sin_t, const int* pos, void* kc, void* vc, const int* base,
                            const int* len, int T, int Hq, int Hk, int D, int table_rows, int* err, cudaStream_t stream);
ELL_API int ell_swiglu_fwd(const void* gu, void* out, int T, int F, cudaStream_t stream);
ELL_API int ell_gemm_thin_route(int T, int N, int K);
ELL_API int ell_gemm_thin(const void* x, const void* W, void* out, const void* bias, int T, int N, int K, int ldx, int ldw, int ldo,
                          int w_mn, int out_mode, int split, int wait_us, int mute, int* err, cudaStream_t stream);
ELL_API int ell_matvec(const void* x, const void* w, const void* bias, void* out, long long xb, long long wb, long long ob, int batch,
                       int M, int N, int K, int ldx, int ldo, int out_f32, int accumulate, int act_tanh, int is_bf16,
                       cudaStream_t stream);
ELL_API int ell_gemm_bf16(const void* A, const void* B, void* C, const void* bias, int M, int N, int K, int lda, int ldb, int ldc,
                          int a_mn, int b_mn, int out_mode, int bn_hint, int* err, cudaStream_t stream);
ELL_API int ell_gemm_bf16_pair(const void* A, const void* B, void* C, const void* bias, int M, int N, int K, int lda, int ldb, int ldc,
                               int a_mn, int b_mn, int out_mode, int* err, cudaStream_t stream);
ELL_API int ell_gemm_pair_route(int M, int N);
ELL_API int ell_gemm_pair_refused(int rc);
ELL_API int ell_gemm_glu_pair(const void* x, const void* W, void* out, const void* bias, int M, int F, int K, int ldx, int ldo, int act,
                              int* err, cudaStream_t stream);
ELL_API int ell_flash_attn_fwd(const void* q, const void* k, const void* v, void* out, float* lse, const int* row_start, int T, int Hq,
                               int Hk, int d, int dv, int q_stride, int k_stride, int v_stride, float scale, const float* alibi_slopes,
                               const float* sink, int window, int* err, cudaStream_t stream);
ELL_API long long ell_attn_rows_scratch(int n, int H, int G, int d, int dv, int max_len, int window, int n_seq, int max_q, int is_bf16);
ELL_API int ell_attn_rows(const void* q, const void* k, const void* v, void* out, float* part, const int* base, const int* len,
                          const float* sink, const float* slopes, const void* gate, int n, int H, int G, int d, int dv, int ldq, int ldk,
                          int ldv, int ldg, int max_len, int window, float scale, const int* cu, int n_seq, int max_q,
                          long long kv_rows, int is_bf16, int* err, cudaStream_t stream);

namespace ell {

// One layer: weights [(Hq + 2 Hk) D, W], [W, Hq D], [2 F, W] (gate first), [W, F], the norms' [W]; the cache's keys and values as kv_rows
// rows of Hk D; rotary tables fp32 [table_rows, D / 2].
struct StepLayer {
  const void *qkv, *o, *gate_up, *down, *norm1, *norm2;
  void *kc, *vc;
  const float *cos, *sin;
  long long table_rows, kv_rows;
};
struct StepArgs {
  const StepLayer* layers;
  const void *x, *norm;           // [T, W]; the weight of the norm behind the layers
  void *y, *work;                 // [T, W]; ell_decoder_step_work bytes, on a 256-byte boundary
  const int *pos, *row_start, *kv_base, *kv_len, *cu;
  int* err;
  long long n_layers, T, W, Hq, Hk, D, F;
  long long fresh;                // prompts that start here: attention within the batch; else over the cached rows
  long long max_len, n_seq, max_q;
  long long gated;                // whether the gated product may run (on CTA pairs)
  long long pairs;                // whether products may run on CTA pairs
  long long launches, failed;     // out: launches; the kind of launch that failed
};
static_assert(sizeof(StepLayer) == 12 * 8 && sizeof(StepArgs) == 26 * 8, "the caller lays them out as 64-bit words");
enum StepPart { kStepNorm = 1, kStepProduct, kStepRotation, kStepAttention, kStepActivation };
// A launch on CTA pairs was refused: the call is repeated without any, or without the gated one alone.
constexpr int kStepNoPairs = -1000, kStepNotGated = -1001;

static bool use_pairs(const StepArgs& a, long long N) { return a.pairs && ell_gemm_pair_route((int)a.T, (int)N); }
static bool use_gated(const StepArgs& a) { return a.gated && use_pairs(a, 2 * a.F); }
static int refused(int rc, int instead) { return ell_gemm_pair_refused(rc) ? instead : rc; }

// out [T, N] = x [T, K] w^T
static int step_product(const StepArgs& a, const void* x, const void* w, void* out, long long N_, long long K_, cudaStream_t stream) {
  const int T = (int)a.T, N = (int)N_, K = (int)K_, route = ell_gemm_thin_route(T, N, K);
  if (route == 2) return ell_matvec(x, w, nullptr, out, 0, 0, 0, 1, T, N, K, K, N, 0, 0, 0, 1, stream);
  if (route) return ell_gemm_thin(x, w, out, nullptr, T, N, K, K, K, N, 0, 0, 0, 0, -1, a.err, stream);
  if (use_pairs(a, N)) return refused(ell_gemm_bf16_pair(x, w, out, nullptr, T, N, K, K, K, N, 0, 0, 0, a.err, stream), kStepNoPairs);
  return ell_gemm_bf16(x, w, out, nullptr, T, N, K, K, K, N, 0, 0, 0, 0, a.err, stream);
}

// Offsets in the work space.  The rows of the attention and those of the feed-forward share their place.
struct StepWork {
  size_t normed, delta, h[2], rstd, qkv, att, lse, part, gate_up, act, bytes;
  bool ranges;                    // the keys of a row are split, so their sums are merged by a second launch
};
static StepWork step_work(const StepArgs& a) {
  StepWork w{};
  size_t at = 0;
  auto take = [&](size_t bytes) {
    const size_t p = at;
    at += (bytes + 255) / 256 * 256;
    return p;
  };
  const size_t T = a.T, row = T * a.W * 2;
  w.normed = take(row);
  w.delta = take(row);
  w.h[0] = take(row);
  w.h[1] = take(row);
  w.rstd = take(T * 4);
  const size_t shared = at;
  w.qkv = take(T * (a.Hq + 2 * a.Hk) * a.D * 2);
  w.att = take(T * a.Hq * a.D * 2);
  if (a.fresh) w.lse = take(T * a.Hq * 4);
  else {
    const long long need = ell_attn_rows_scratch((int)T, (int)a.Hq, (int)a.Hk, (int)a.D, (int)a.D, (int)a.max_len, 0, (int)a.n_seq,
                                                 (int)a.max_q, 1);
    w.ranges = need > 0;
    w.part = take((size_t)need * 4);
  }
  const size_t end = at;
  at = shared;
  w.act = take(T * a.F * 2);
  if (!use_gated(a)) w.gate_up = take(T * 2 * a.F * 2);
  w.bytes = std::max(at, end);
  return w;
}

static int step_layers(StepArgs& a, float eps, float scale, cudaStream_t stream) {
  const StepWork at = step_work(a);
  const int T = (int)a.T, W = (int)a.W, Hq = (int)a.Hq, Hk = (int)a.Hk, D = (int)a.D, F = (int)a.F, ld = (Hq + 2 * Hk) * D;
  char* work = static_cast<char*>(a.work);
  void *normed = work + at.normed, *delta = work + at.delta, *att = work + at.att, *act = work + at.act, *gate_up = work + at.gate_up;
  __nv_bfloat16* qkv = reinterpret_cast<__nv_bfloat16*>(work + at.qkv);
  float *rstd = reinterpret_cast<float*>(work + at.rstd), *part = reinterpret_cast<float*>(work + at.part);
  // the residual stream: the input, then one of two buffers, which the next sum leaves for the other
  const void *h = nullptr, *d = a.x;
  int turn = 0, rc;
  auto add_norm = [&](const void* weight, void* y) {
    void* to = work + at.h[turn];
    const int r = ell_rmsnorm_fwd(d, h, weight, y, h ? to : nullptr, rstd, T, W, eps, stream);
    if (h) turn ^= 1;
    h = h ? to : d;
    return r;
  };
#define ELL_STEP(part_, call)                                 \
  if ((rc = (call)) != 0) return a.failed = part_, rc;        \
  ++a.launches
  for (long long i = 0; i < a.n_layers; ++i) {
    const StepLayer& l = a.layers[i];
    ELL_STEP(kStepNorm, add_norm(l.norm1, normed));
    ELL_STEP(kStepProduct, step_product(a, normed, l.qkv, qkv, ld, W, stream));
    ELL_STEP(kStepRotation, ell_rope_append(qkv, l.cos, l.sin, a.pos, l.kc, l.vc, a.kv_base, a.kv_len, T, Hq, Hk, D, (int)l.table_rows,
                                            a.err, stream));
    if (a.fresh) {
      ELL_STEP(kStepAttention, ell_flash_attn_fwd(qkv, qkv + Hq * D, qkv + (Hq + Hk) * D, att, reinterpret_cast<float*>(work + at.lse),
                                                  a.row_start, T, Hq, Hk, D, D, ld, ld, ld, scale, nullptr, nullptr, 0, a.err, stream));
    } else {
      ELL_STEP(kStepAttention, ell_attn_rows(qkv, l.kc, l.vc, att, at.ranges ? part : nullptr, a.kv_base, a.kv_len, nullptr, nullptr, nullptr, T, Hq, Hk, D, D,
                                             ld, Hk * D, Hk * D, 0, (int)a.max_len, 0, scale, a.n_seq ? a.cu : nullptr, (int)a.n_seq,
                                             (int)a.max_q, l.kv_rows, 1, a.err, stream));
      a.launches += at.ranges;
    }
    ELL_STEP(kStepProduct, step_product(a, att, l.o, delta, W, Hq * D, stream));
    d = delta;
    ELL_STEP(kStepNorm, add_norm(l.norm2, normed));
    if (use_gated(a)) {
      ELL_STEP(kStepProduct, refused(ell_gemm_glu_pair(normed, l.gate_up, act, nullptr, T, F, W, W, F, 1, a.err, stream), kStepNotGated));
    } else {
      ELL_STEP(kStepProduct, step_product(a, normed, l.gate_up, gate_up, 2 * F, W, stream));
      ELL_STEP(kStepActivation, ell_swiglu_fwd(gate_up, act, T, F, stream));
    }
    ELL_STEP(kStepProduct, step_product(a, act, l.down, delta, W, F, stream));
  }
  ELL_STEP(kStepNorm, add_norm(a.norm, a.y));
#undef ELL_STEP
  return 0;
}

}  // namespace ell

using namespace ell;

// Bytes of work space of a call.
ELL_API long long ell_decoder_step_work(const long long* args) {
  return (long long)step_work(*reinterpret_cast<const StepArgs*>(args)).bytes;
}

// The normed rows y behind `n_layers` layers (norm, attention, norm, gated feed-forward; residual sums in bf16) for the T new rows x of
// a step, whose keys and values go to the caches.  D a multiple of 16 up to 128, W and F multiples of 8, all on 16-byte boundaries.
// args: the words of StepArgs.  kStepNoPairs, kStepNotGated: to be called again with `pairs`, or `gated`, 0 (what it has written so far is
// written again).
ELL_API int ell_decoder_step(long long* args, float eps, float scale, cudaStream_t stream) {
  StepArgs& a = *reinterpret_cast<StepArgs*>(args);
  a.launches = a.failed = 0;
  if (a.T <= 0) return 0;
  if (a.n_layers < 1 || a.D % 16 || a.D > 128 || a.W % 8 || a.F % 8 || !aligned_to(a.work, 256)) return -2;
  return step_layers(a, eps, scale, stream);
}
