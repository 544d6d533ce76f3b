// The launches of one transformer block's forward and of its backward as one host call each. The block (ops/block.py) is a
// straight line of 14 to 20 launches in the forward and about 25 in the backward; issued one by one from Python each costs
// 15 to 25 us of interpreter and ctypes time, more than the kernels of a small model run for. Here the caller fills one
// argument struct (the tensors are allocated by the framework as before) and the launchers follow one another in C++.
//
// Both functions return the number of launchers called, or -(1000 * step + code) when the launcher of that step refused its
// arguments with -code; nothing is launched after that. Pass of a 4-layer
// model of d = 256, bound by the host: 6.1 -> 3.7 ms; prompt logits of a 16-layer model of d = 1024: 10.3 -> 4.8 ms.
#include <cuda_runtime.h>
#include <stdint.h>

typedef const void* cptr;
typedef const float* cf;
extern "C" {
int sr_gemm_bf16(cptr A, cptr B, void* C, cptr Cin, int M, int N, int K, int batch, long long lda, long long ldb, long long ldc,
                 long long ldcin, long long strideA, long long strideB, long long strideC, long long strideCin, int a_mn, int b_mn,
                 int c_fp32, int cin_fp32, float alpha, float beta, cf alpha_ptr, cf row_scale, int sym, int bn, int max_ctas,
                 int* status, cudaStream_t stream);
int sr_rmsnorm_fwd(cptr x, void* y, long rows, int D, long ldx, float eps, cudaStream_t s);
int sr_rmsnorm_bwd(cptr x, cptr dy, cptr dres, void* dx, long rows, int D, long ldx, float eps, cudaStream_t s);
int sr_mix_norm_fwd(cptr xp, cptr x0, cptr skip, void* x, void* a, cf lr, cf l0, cf ws, long rows, int D, float eps, cudaStream_t s);
int sr_norm_bwd_mix(cptr x, cptr da, cptr g_res, cptr g_res2, cptr xp, cptr x0, cptr skip, void* dxp, void* dx0, void* dskip, cf lr,
                    cf l0, cf ws, float* d_lr, float* d_l0, float* d_ws, long rows, int D, float eps, cudaStream_t s);
int sr_iha_mix_fwd(cf mix, cptr W, void* out, int P, int H, long J, cudaStream_t s);
int sr_iha_mix_bwd(cf mix, cptr W, cptr dWp, float* gradW, float* dmix, int P, int H, long J, cudaStream_t s);
int sr_gate_fwd(cptr a, long lda, cf W, float* gate, long M, int H, int nc, float scale, cudaStream_t s);
int sr_gate_bwd(cf dgate, cf gate, cptr a, long lda, cf W, float* dW, void* da, long ldda, long M, int H, int nc, float scale,
                cudaStream_t s);
int sr_qkv_prep_fwd(cptr qkv, cptr ve, cf gate, cptr cosb, cptr sinb, void* q, void* k, void* v, long tokens, int H, int T, float eps,
                    int key_offset, cudaStream_t s);
int sr_qkv_prep_bwd_f32dq(cptr qkv, cptr ve, cf gate, cptr cosb, cptr sinb, cf dq_f32, cptr dk, cptr dv, void* dqkv, void* dve,
                          float* dgate, long tokens, int H, int T, float eps, int key_offset, cptr dv_extra, cudaStream_t s);
int sr_flash_attn_fwd(cptr q, cptr k, cptr v, void* out, float* lse, int B, int T, int H, long ld_q, long ld_k, long ld_v, int window,
                      float scale, int bkv, int* status, cudaStream_t stream);
int sr_flash_attn_bwd_ex(cptr dO, cptr q, cptr k, cptr v, cptr out, cf lse, float* delta, float* dq_acc, void* dq, void* dk, void* dv,
                         int B, int T, int H, int window, float scale, int flags, int* status, cudaStream_t stream);
int sr_attn_post_fwd(cptr y, cptr v, cf gate, cf alpha, void* out, long tokens, int H, float xsa_eps, cudaStream_t s);
int sr_attn_post_bwd(cptr g, cptr y, cptr v, cf gate, cf alpha, void* dy, float* dgate, float* delta, void* dv_x, float* dalpha,
                     long tokens, int H, int T, float xsa_eps, cudaStream_t s);
int sr_add_norm_fwd(cptr x, cptr y, void* x_mid, void* n, long rows, int D, float eps, float p, unsigned long long seed,
                    const unsigned long long* seed_ptr, cudaStream_t s);
int sr_norm_bwd_drop(cptr x_mid, cptr dn, cptr g_res, void* dx_mid, void* dy, long rows, int D, float eps, float p,
                     unsigned long long seed, const unsigned long long* seed_ptr, cudaStream_t s);
int sr_swiglu_fwd(cptr gf, void* out, long M, int h, cudaStream_t s);
int sr_swiglu_bwd(cptr gf, cptr dout, void* dgf, long M, int h, cudaStream_t s);
int sr_dropout_add_fwd(cptr x_mid, cptr y, cptr x_in, cf keep, void* out, long n, float p, unsigned long long seed,
                       const unsigned long long* seed_ptr, cudaStream_t s);
int sr_dropout_add_bwd(cptr g, cf keep, void* dy, void* dmid, void* din, long n, float p, unsigned long long seed,
                       const unsigned long long* seed_ptr, cudaStream_t s);
}

// Mirrored field by field in ops/block.py (_Shape, _FwdArgs, _BwdArgs). All matrices are row-major and dense: activations
// [M, C], [M, 3C], [M, 2 hdim], weights [out, in]; null = the block has no such part.
struct BlockShape {
  long long M;                                  // tokens = B * T
  int B, T, C, H, hdim, window, key_offset, do_mix, attn_bkv, gate_nc, ve_gate_nc;
  float eps, xsa_eps, scale, p_attn, p_mlp;
  unsigned long long seed1, seed2;
  const unsigned long long* drop_state;
  int* status;
  // weights and per-layer scalars
  cf rl, xl, sw;                                // lambda mix
  cptr ve_w;
  cf mixes;                                     // [3, H, H]
  cptr qkv_w;
  cf gate_w, ve_gate_w;
  cptr cosb, sinb;
  cf xsa;                                       // [H]
  cptr proj_w, gf_w, mo_w;
};
struct BlockFwd {
  BlockShape s;
  cptr xp, x0, sk;
  void *x, *a, *ve, *w_mix, *qkv;
  float *agate, *ve_gate;
  void *q, *k, *v, *y;
  float* lse;
  void *y2, *o, *x_mid, *n, *gf, *hdn, *mo;
  cf keep;
  void* out;
};
struct BlockBwd {
  BlockShape s;
  cptr g, xp, x0, sk;
  // saved by the forward
  cptr x, a, ve, w_qkv, qkv;
  cf agate, ve_gate;
  cptr q, k, v, y;
  cf lse;
  cptr y2, x_mid, n, gf, hdn;
  cf keep;
  // temporaries
  void *dmo, *g_mid, *g_in, *dhdn, *dgf, *dn, *g_mid_tot, *d_o, *dy2, *dy;
  float *dagate, *delta;
  void* dv_x;
  float* dq;
  void *dk, *dv, *dqkv, *dve;
  float* dvegate;
  void *da, *dwp;
  // results
  void *dxp, *dx0, *dsk;
  float *g_mo, *g_gf, *g_proj, *g_qkv, *g_mix, *g_gate, *g_ve_gate, *g_ve, *g_rl, *g_xl, *g_sw, *g_xsa;
};

namespace {

// out = A B^T (b_mn: A B) with dense operands; acc: out (fp32, or bf16 with out_bf16) += the product; a_mn: A^T
struct Gemm {
  int* status;
  cudaStream_t st;
  // activations: [M, K] x weight
  int fwd(cptr x, cptr w, void* out, long long M, int N, int K) const {          // w [N, K]
    return sr_gemm_bf16(x, w, out, nullptr, (int)M, N, K, 1, K, K, N, 0, 0, 0, 0, 0, 0, 0, 0, 0, 1.f, 0.f, nullptr, nullptr, 0, 0, 0, status, st);
  }
  int dx(cptr g, cptr w, void* out, long long M, int N, int K, bool add = false) const {   // w [K, N]: out [M, N] (+)= g [M, K] w
    return sr_gemm_bf16(g, w, out, add ? out : nullptr, (int)M, N, K, 1, K, N, N, add ? N : 0, 0, 0, 0, 0, 0, 1, 0, 0, 1.f,
                        add ? 1.f : 0.f, nullptr, nullptr, 0, 0, 0, status, st);
  }
  int dw(cptr g, cptr x, float* grad, long long M, int N, int K) const {          // grad [N, K] += g^T [N, M] x [M, K]
    return sr_gemm_bf16(g, x, grad, grad, N, K, (int)M, 1, N, K, K, K, 0, 0, 0, 0, 1, 1, 1, 1, 1.f, 1.f, nullptr, nullptr, 0, 0, 0, status, st);
  }
  int dw_bf16(cptr g, cptr x, void* out, long long M, int N, int K) const {
    return sr_gemm_bf16(g, x, out, nullptr, N, K, (int)M, 1, N, K, K, 0, 0, 0, 0, 0, 1, 1, 0, 0, 1.f, 0.f, nullptr, nullptr, 0, 0, 0, status, st);
  }
};

}  // namespace

#define STEP(call)                                        \
  do {                                                    \
    ++step;                                               \
    if (int rc_ = (call)) return -(1000 * step + (rc_ < 0 ? -rc_ : rc_)); \
  } while (0)

extern "C" int sr_block_fwd(const BlockFwd* p, cudaStream_t st) {
  const BlockShape& s = p->s;
  const Gemm gemm{s.status, st};
  const long M = (long)s.M, J = 128L * s.C;
  int step = 0;
  if (s.do_mix) STEP(sr_mix_norm_fwd(p->xp, p->x0, p->sk, p->x, p->a, s.rl, s.xl, s.sw, M, s.C, s.eps, st));
  else          STEP(sr_rmsnorm_fwd(p->x, p->a, M, s.C, s.C, s.eps, st));
  if (s.ve_w) STEP(gemm.fwd(p->x0, s.ve_w, p->ve, M, s.C, s.C));
  if (s.mixes) STEP(sr_iha_mix_fwd(s.mixes, s.qkv_w, p->w_mix, 3, s.H, J, st));
  STEP(gemm.fwd(p->a, s.mixes ? p->w_mix : s.qkv_w, p->qkv, M, 3 * s.C, s.C));
  STEP(sr_gate_fwd(p->a, s.C, s.gate_w, p->agate, M, s.H, s.gate_nc, 1.f, st));
  if (s.ve_w) STEP(sr_gate_fwd(p->a, s.C, s.ve_gate_w, p->ve_gate, M, s.H, s.ve_gate_nc, 2.f, st));
  STEP(sr_qkv_prep_fwd(p->qkv, p->ve, p->ve_gate, s.cosb, s.sinb, p->q, p->k, p->v, M, s.H, s.T, s.eps, s.key_offset, st));
  STEP(sr_flash_attn_fwd(p->q, p->k, p->v, p->y, p->lse, s.B, s.T, s.H, s.C, s.C, s.C, s.window, s.scale, s.attn_bkv, s.status, st));
  STEP(sr_attn_post_fwd(p->y, p->v, p->agate, s.xsa, p->y2, M, s.H, s.xsa_eps, st));
  STEP(gemm.fwd(p->y2, s.proj_w, p->o, M, s.C, s.C));
  STEP(sr_add_norm_fwd(p->x, p->o, p->x_mid, p->n, M, s.C, s.eps, s.p_attn, s.seed1, s.drop_state, st));
  STEP(gemm.fwd(p->n, s.gf_w, p->gf, M, 2 * s.hdim, s.C));
  STEP(sr_swiglu_fwd(p->gf, p->hdn, M, s.hdim, st));
  STEP(gemm.fwd(p->hdn, s.mo_w, p->mo, M, s.C, s.hdim));
  STEP(sr_dropout_add_fwd(p->x_mid, p->mo, p->keep ? p->x : nullptr, p->keep, p->out, M * s.C, s.p_mlp, s.seed2, s.drop_state, st));
  return step;
}

extern "C" int sr_block_bwd(const BlockBwd* p, cudaStream_t st) {
  const BlockShape& s = p->s;
  const Gemm gemm{s.status, st};
  const long M = (long)s.M, J = 128L * s.C;
  int step = 0;
  // MLP branch
  STEP(sr_dropout_add_bwd(p->g, p->keep, p->dmo, p->g_mid, p->g_in, M * s.C, s.p_mlp, s.seed2, s.drop_state, st));
  const cptr g_mid = p->keep ? p->g_mid : p->g;
  STEP(gemm.dx(p->dmo, s.mo_w, p->dhdn, M, s.hdim, s.C));
  STEP(gemm.dw(p->dmo, p->hdn, p->g_mo, M, s.C, s.hdim));
  STEP(sr_swiglu_bwd(p->gf, p->dhdn, p->dgf, M, s.hdim, st));
  STEP(gemm.dx(p->dgf, s.gf_w, p->dn, M, s.C, 2 * s.hdim));
  STEP(gemm.dw(p->dgf, p->n, p->g_gf, M, 2 * s.hdim, s.C));
  // attention branch
  STEP(sr_norm_bwd_drop(p->x_mid, p->dn, g_mid, p->g_mid_tot, p->d_o, M, s.C, s.eps, s.p_attn, s.seed1, s.drop_state, st));
  STEP(gemm.dx(p->d_o, s.proj_w, p->dy2, M, s.C, s.C));
  STEP(gemm.dw(p->d_o, p->y2, p->g_proj, M, s.C, s.C));
  STEP(sr_attn_post_bwd(p->dy2, p->y, p->v, p->agate, s.xsa, p->dy, p->dagate, p->delta, p->dv_x, p->g_xsa, M, s.H, s.T, s.xsa_eps, st));
  STEP(cudaMemsetAsync(p->dq, 0, (size_t)M * s.C * sizeof(float), st) == cudaSuccess ? 0 : -5);
  STEP(sr_flash_attn_bwd_ex(p->dy, p->q, p->k, p->v, p->y, p->lse, p->delta, p->dq, nullptr, p->dk, p->dv, s.B, s.T, s.H, s.window,
                            s.scale, 3, s.status, st));      // delta given, dQ stays fp32
  STEP(sr_qkv_prep_bwd_f32dq(p->qkv, p->ve, p->ve_gate, s.cosb, s.sinb, p->dq, p->dk, p->dv, p->dqkv, p->dve, p->dvegate, M, s.H, s.T,
                             s.eps, s.key_offset, p->dv_x, st));
  STEP(gemm.dx(p->dqkv, p->w_qkv, p->da, M, s.C, 3 * s.C));
  if (s.mixes) {
    STEP(gemm.dw_bf16(p->dqkv, p->a, p->dwp, M, 3 * s.C, s.C));
    STEP(sr_iha_mix_bwd(s.mixes, s.qkv_w, p->dwp, p->g_qkv, nullptr, 3, s.H, J, st));
    // dmix[p] += dW'[p] W[p]^T, [H x J] x [J x H]
    const long long HJ = (long long)s.H * J, HH = (long long)s.H * s.H;
    STEP(sr_gemm_bf16(p->dwp, s.qkv_w, p->g_mix, p->g_mix, s.H, s.H, (int)J, 3, J, J, s.H, s.H, HJ, HJ, HH, HH, 0, 0, 1, 1, 1.f, 1.f,
                      nullptr, nullptr, 0, 128, 0, s.status, st));
  } else {
    STEP(gemm.dw(p->dqkv, p->a, p->g_qkv, M, 3 * s.C, s.C));
  }
  STEP(sr_gate_bwd(p->dagate, p->agate, p->a, s.C, s.gate_w, p->g_gate, p->da, s.C, M, s.H, s.gate_nc, 1.f, st));
  if (s.ve_w) {
    STEP(sr_gate_bwd(p->dvegate, p->ve_gate, p->a, s.C, s.ve_gate_w, p->g_ve_gate, p->da, s.C, M, s.H, s.ve_gate_nc, 2.f, st));
    STEP(gemm.dw(p->dve, p->x0, p->g_ve, M, s.C, s.C));
  }
  if (s.do_mix) {
    STEP(sr_norm_bwd_mix(p->x, p->da, p->g_mid_tot, p->g_in, p->xp, p->x0, p->sk, p->dxp, p->dx0, p->dsk, s.rl, s.xl, s.sw, p->g_rl,
                         p->g_xl, p->g_sw, M, s.C, s.eps, st));
    if (s.ve_w) STEP(gemm.dx(p->dve, s.ve_w, p->dx0, M, s.C, s.C, true));
  } else {
    STEP(sr_rmsnorm_bwd(p->x, p->da, p->g_mid_tot, p->dxp, M, s.C, s.C, s.eps, st));
    if (s.ve_w) STEP(gemm.dx(p->dve, s.ve_w, p->dx0, M, s.C, s.C));
  }
  return step;
}
