// One transformer block, forward and backward, as the sequence of launches that its operators make one by one: a training
// step of a small model is bound by the host, which spends several times longer per operator on Python than on its launches.
// The forward makes the launches of ml_framework_b200/ops/functional.py, in their order. The backward's are the same products,
// attention and normalisation kernels with the same arguments; the bias gradients of two products share a launch, behind both
// products' weight gradients, and have the row split of that launch.
//
//   forward   h1 = norm(x); qkv = h1 Wqkv^T (+ b); [rotary embedding in place]; a = attention(qkv); x1 = x + a Wo^T (+ b);
//             h2 = norm(x1); act = f(h2 W1^T (+ b)), pre = its argument; y = x1 + act W2^T (+ b)
//   backward  the gradients of x and of every parameter, the latter into their buffers (written or, by a bit of `accumulate`
//             each, added)
// gated = 0: layer norm, biases, tanh-GELU; gated = 1: RMS norm, rotary embedding, SwiGLU over interleaved gate / up rows.
//
// A step of two layers of 256 on 2 x 256 tokens, whose kernels take 0.4 ms: 1.88 ms operator by operator, 0.88 ms like this
// (0.24 ms of the gain because the engine no longer hands the backward to autograd's device thread).
#include "../common/host.h"
#include "../mlf_api.h"

using namespace mlf;

extern "C" {
int mlf_norm_fwd(const void* x, const void* gamma, const void* beta, void* y, float* mean, float* rstd, int rows, int D, float eps, int rms,
                 uint64_t stream);
int mlf_norm_bwd_add(const void* x, const void* dy, const void* gamma, const float* mean, const float* rstd, void* dx, void* dgamma, void* dbeta,
                     float* partials, int rows, int D, int rms, int grads_fp32, int accumulate_gamma, int accumulate_beta, const void* dx_add,
                     uint64_t stream);
int mlf_rope_qkv(void* out, const void* in, const long long* pos, long long T, int Hq, int Hkv, long long ldo, long long ldi, float theta,
                 int inverse, uint64_t stream);
int mlf_flash_fwd(const void* q, const void* k, const void* v, void* out, float* lse, int B, int S, int Hq, int Hkv, long long ldq, long long ldk,
                  long long ldv, long long ldo, float scale, int causal, uint64_t stream);
int mlf_flash_bwd(const void* q, const void* k, const void* v, const void* o, const void* dout, const float* lse, void* dq, void* dk, void* dv,
                  void* scratch, int B, int S, int Hq, int Hkv, long long ldq, long long ldk, long long ldv, long long ldo, long long lddo,
                  long long lddq, long long lddk, long long lddv, float scale, int causal, uint64_t stream);
int mlf_colsum2(void* db0, const void* dy0, int N0, long long ld0, int accumulate0, void* db1, const void* dy1, int N1, long long ld1,
                int accumulate1, int M, void* scratch, uint64_t stream);
}

namespace {

// out = epilogue(A B^T); operands K-major unless a_mn / b_mn
int product(const void* a, const void* b, void* out, int M, int N, int K, int lda, int ldb, int ldo, int a_mn, int b_mn, int flags,
            const void* bias, const void* aux_in, int ld_aux_in, void* aux_out, int ld_aux_out, uint64_t stream) {
  MlfGemmArgs g = {};
  g.a = a; g.b = b; g.out = out; g.bias = bias; g.aux_in = aux_in; g.aux_out = aux_out;
  g.M = M; g.N = N; g.K = K; g.lda = lda; g.ldb = ldb; g.ldo = ldo; g.ld_aux_in = ld_aux_in; g.ld_aux_out = ld_aux_out;
  g.a_mn = a_mn; g.b_mn = b_mn;
  g.flags = flags | (bias != nullptr ? MLF_EPI_BIAS : 0);
  g.alpha = 1.f;
  return mlf_gemm_bf16(&g, stream);
}

const char* at(const void* p, long long elems) { return static_cast<const char*>(p) + 2 * elems; }
char* at(void* p, long long elems) { return static_cast<char*>(p) + 2 * elems; }

}  // namespace

#define RUN(call)            \
  do {                       \
    const int _rc = (call);  \
    if (_rc) return _rc;     \
  } while (0)

static int check_block(const MlfBlockArgs* p) {
  MLF_REQUIRE(p != nullptr && p->B > 0 && p->S > 0 && p->d > 0 && p->ff > 0 && p->Hq > 0 && p->Hkv > 0 && p->Hq % p->Hkv == 0, "block: bad shape");
  return 0;
}

MLF_API int mlf_block_forward(const MlfBlockArgs* p, uint64_t st) {
  RUN(check_block(p));
  const int T = p->B * p->S, d = p->d, q = p->Hq * 128, kv = p->Hkv * 128, w = q + 2 * kv, n1 = p->gated ? 2 * p->ff : p->ff;
  RUN(mlf_norm_fwd(p->x, p->g1, p->b1, p->h1, p->mean1, p->rstd1, T, d, p->eps1, p->gated, st));
  RUN(product(p->h1, p->wqkv, p->qkv, T, w, d, d, d, w, 0, 0, 0, p->bqkv, nullptr, 0, nullptr, 0, st));
  if (p->pos != nullptr) RUN(mlf_rope_qkv(p->qkv, p->qkv, p->pos, T, p->Hq, p->Hkv, w, w, p->rope_theta, 0, st));
  RUN(mlf_flash_fwd(p->qkv, at(p->qkv, q), at(p->qkv, q + kv), p->a, p->lse, p->B, p->S, p->Hq, p->Hkv, w, w, w, q, p->scale, p->causal, st));
  RUN(product(p->a, p->wo, p->x1, T, d, q, q, q, d, 0, 0, MLF_EPI_RESIDUAL, p->bo, p->x, d, nullptr, 0, st));
  RUN(mlf_norm_fwd(p->x1, p->g2, p->b2, p->h2, p->mean2, p->rstd2, T, d, p->eps2, p->gated, st));
  RUN(product(p->h2, p->w1, p->act, T, n1, d, d, d, p->ff, 0, 0, (p->gated ? MLF_EPI_SWIGLU : MLF_EPI_GELU) | MLF_EPI_STORE_PRE, p->bb1, nullptr, 0,
              p->pre, n1, st));
  return product(p->act, p->w2, p->y, T, d, p->ff, p->ff, p->ff, d, 0, 0, MLF_EPI_RESIDUAL, p->bb2, p->x1, d, nullptr, 0, st);
}

MLF_API int mlf_block_backward(const MlfBlockArgs* p, uint64_t st) {
  RUN(check_block(p));
  const int T = p->B * p->S, d = p->d, q = p->Hq * 128, kv = p->Hkv * 128, w = q + 2 * kv, n1 = p->gated ? 2 * p->ff : p->ff;
  auto add = [&](int bit) { return (p->accumulate >> bit) & 1; };
  // dW [out, in] = dy^T x
  auto wgrad = [&](const void* dy, const void* x, void* dw, int out, int in, int bit) {
    return product(dy, x, dw, out, in, T, out, in, in, 1, 1, add(bit) ? MLF_EPI_ACCUM : 0, nullptr, nullptr, 0, nullptr, 0, st);
  };
  // Bias gradients of two products, the column sums of their dY. Layer-norm blocks have all of them, gated ones none.
  auto bgrads = [&](const void* dy0, void* db0, int bit0, const void* dy1, void* db1, int width1, int bit1) {
    return db0 == nullptr ? 0 : mlf_colsum2(db0, dy0, d, d, add(bit0), db1, dy1, width1, width1, add(bit1), T, p->colsum_scratch, st);
  };
  // MLP: dpre, then dh2
  RUN(product(p->dy, p->w2, p->wide, T, p->ff, d, d, p->ff, n1, 0, 1, p->gated ? MLF_EPI_DSWIGLU : MLF_EPI_DGELU_MUL, nullptr, p->pre, n1, nullptr, 0, st));
  RUN(wgrad(p->dy, p->act, p->dw2, d, p->ff, MLF_BLOCK_W2));
  RUN(wgrad(p->wide, p->h2, p->dw1, n1, d, MLF_BLOCK_W1));
  RUN(bgrads(p->dy, p->dbb2, MLF_BLOCK_BB2, p->wide, p->dbb1, n1, MLF_BLOCK_BB1));
  RUN(product(p->wide, p->w1, p->row, T, d, n1, n1, d, d, 0, 1, 0, nullptr, nullptr, 0, nullptr, 0, st));
  RUN(mlf_norm_bwd_add(p->x1, p->row, p->g2, p->mean2, p->rstd2, p->dx1, p->dg2, p->db2, p->norm_scratch, T, d, p->gated, 0, add(MLF_BLOCK_G2),
                       add(MLF_BLOCK_B2), p->dy, st));
  // attention: da, dqkv (in the MLP's place), then dh1
  RUN(product(p->dx1, p->wo, p->da, T, q, d, d, q, q, 0, 1, 0, nullptr, nullptr, 0, nullptr, 0, st));
  RUN(wgrad(p->dx1, p->a, p->dwo, d, q, MLF_BLOCK_WO));
  RUN(mlf_flash_bwd(p->qkv, at(p->qkv, q), at(p->qkv, q + kv), p->a, p->da, p->lse, p->wide, at(p->wide, q), at(p->wide, q + kv), p->flash_scratch,
                    p->B, p->S, p->Hq, p->Hkv, w, w, w, q, q, w, w, w, p->scale, p->causal, st));
  if (p->pos != nullptr) RUN(mlf_rope_qkv(p->wide, p->wide, p->pos, T, p->Hq, p->Hkv, w, w, p->rope_theta, 1, st));
  RUN(product(p->wide, p->wqkv, p->row, T, d, w, w, d, d, 0, 1, 0, nullptr, nullptr, 0, nullptr, 0, st));
  RUN(wgrad(p->wide, p->h1, p->dwqkv, w, d, MLF_BLOCK_WQKV));
  RUN(bgrads(p->dx1, p->dbo, MLF_BLOCK_BO, p->wide, p->dbqkv, w, MLF_BLOCK_BQKV));
  return mlf_norm_bwd_add(p->x, p->row, p->g1, p->mean1, p->rstd1, p->dx, p->dg1, p->db1, p->norm_scratch, T, d, p->gated, 0, add(MLF_BLOCK_G1),
                          add(MLF_BLOCK_B1), p->dx1, st);
}
