"""GPU tests of kernel variants at the sizes where they change: tile edges, remainders, the ends of their ranges."""
import itertools

import pytest
import torch

pytestmark = pytest.mark.gpu


def _status_ok():
    from slowrun_b200.ops import _lib
    torch.cuda.synchronize()
    _lib.check_status()


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm()).item()


# --------------------------------------------------------------------------------------------- GEMM output paths
@pytest.mark.parametrize("M,N,K,batch", [(129, 8, 64, 1), (257, 264, 72, 1), (300, 1000, 200, 1), (1920, 640, 3000, 1),
                                         (513, 136, 320, 3), (700, 33, 128, 1), (260, 257, 136, 1)])
@pytest.mark.parametrize("pad", [0, 3, 8])
def test_gemm_output_boxes_stay_inside_the_matrix(M, N, K, batch, pad):
    """bf16 and fp32 stores and fp32 accumulation in place, into a view whose surroundings must not change. Errors: operands
    are exact in fp32, so what is left is fp32 summation (2^-24 sqrt(K) is 4e-6 at most) and the rounding of a bf16 result
    (2^-9)."""
    from slowrun_b200.ops.gemm import gemm, gemm_reference
    g = torch.Generator(device="cuda").manual_seed(M + N)
    r8 = lambda n: (n + 7) // 8 * 8
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    for a_mn, b_mn in itertools.product((False, True), repeat=2):
        A = rnd(batch, K, r8(M))[..., :M] if a_mn else rnd(batch, M, r8(K))[..., :K]
        B = rnd(batch, K, r8(N))[..., :N] if b_mn else rnd(batch, N, r8(K))[..., :K]
        ref = gemm_reference(A.double().bfloat16(), B, a_mn=a_mn, b_mn=b_mn, out_dtype=torch.float32)
        for dt, tol in ((torch.bfloat16, 4e-3), (torch.float32, 1e-5)):
            big = torch.full((batch, M + 2, N + pad), 7.0, device="cuda", dtype=dt)
            gemm(A, B, out=big[:, :M, :N], a_mn=a_mn, b_mn=b_mn)
            _status_ok()
            assert _rel(big[:, :M, :N], ref) < tol
            assert bool((big[:, M:] == 7).all()) and bool((big[:, :, N:] == 7).all())
        c0 = torch.randn(batch, M + 2, N + pad, device="cuda", generator=g)
        big = c0.clone()
        out = big[:, :M, :N]
        gemm(A, B, out=out, cin=out, beta=1.0, a_mn=a_mn, b_mn=b_mn)
        _status_ok()
        assert _rel(out, ref + c0[:, :M, :N]) < 1e-5
        assert torch.equal(big[:, M:], c0[:, M:]) and torch.equal(big[:, :, N:], c0[:, :, N:])


# --------------------------------------------------------------------------------------------- attention
def _attention64(q, k, v, do, window, scale):
    q, k, v = (t.double().detach().requires_grad_() for t in (q, k, v))
    T = q.size(1)
    s = torch.einsum("bqhd,bkhd->bhqk", q, k) * scale
    i = torch.arange(T, device=q.device)
    m = i[None, :] <= i[:, None]
    if window >= 0:
        m &= i[None, :] >= i[:, None] - window
    s = s.masked_fill(~m, float("-inf"))
    o = torch.einsum("bhqk,bkhd->bqhd", s.softmax(-1), v)
    o.backward(do.double())
    return o.detach(), torch.logsumexp(s, -1).detach(), q.grad, k.grad, v.grad


@pytest.mark.parametrize("bkv", [None, 64, 128])
@pytest.mark.parametrize("B,T,H,window", [(1, 5, 2, -1), (3, 129, 1, 128), (1, 130, 1, 3), (1, 256, 2, -1), (1, 257, 1, 200),
                                          (1, 777, 2, 127), (1, 777, 2, 128), (1, 513, 2, 255), (2, 1000, 3, -1),
                                          (1, 1300, 2, 512)])
def test_attention_tile_edges(B, T, H, window, bkv):
    """Forward variants and the backward against fp64. bf16 operands of the products and bf16 results: 2^-9 relative per
    rounding, a few of which meet in dQ and dK."""
    from slowrun_b200.ops.flash_attention import native_bwd, native_fwd
    g = torch.Generator(device="cuda").manual_seed(T + window)
    q, k, v, do = (torch.randn(B, T, H, 128, device="cuda", generator=g).bfloat16() for _ in range(4))
    o, lse, sc, w = native_fwd(q, k, v, window, 0.12, bkv=bkv)
    dq, dk, dv = native_bwd(do, q, k, v, o, lse, sc, w, dq_fp32=True)
    _status_ok()
    ro, rl, rq, rk, rv = _attention64(q, k, v, do, window, 0.12)
    assert _rel(o, ro) < 4e-3 and (lse - rl).abs().max().item() < 1e-2
    assert _rel(dv, rv) < 5e-3
    assert _rel(dq, rq) < 1.2e-2 and _rel(dk, rk) < 1.2e-2


# --------------------------------------------------------------------------------------------- IHA mixing
@pytest.mark.parametrize("H", [1, 3, 5, 12, 19, 21, 32])
def test_iha_mixing_for_every_head_count(H):
    from slowrun_b200.ops.block import iha_mix_backward, iha_mix_weights
    P, J = 3, 128 * H + 8
    g = torch.Generator(device="cuda").manual_seed(H)
    mixes = (torch.eye(H, device="cuda") + 0.1 * torch.randn(P, H, H, device="cuda", generator=g)).contiguous()
    w = (0.05 * torch.randn(P * H, J, device="cuda", generator=g)).bfloat16()
    dwp = (0.01 * torch.randn(P * H, J, device="cuda", generator=g)).bfloat16()
    m64, w64, d64 = mixes.bfloat16().double(), w.view(P, H, J).double(), dwp.view(P, H, J).double()
    out = iha_mix_weights(mixes, w, H)
    assert _rel(out.view(P, H, J), m64 @ w64) < 4e-3                       # one bf16 rounding
    gw = torch.randn(P * H, J, device="cuda", generator=g)
    want = gw.view(P, H, J).double() + m64.transpose(1, 2) @ d64
    acc = torch.zeros(P, H, H, device="cuda")
    assert iha_mix_backward(mixes, w, dwp, gw, H, acc) is None
    _status_ok()
    assert _rel(gw.view(P, H, J), want) < 1e-6
    assert _rel(acc, d64 @ w64.transpose(1, 2)) < 1e-5                     # fp32 sums over J


# --------------------------------------------------------------------------------------------- gated delta rule
@pytest.mark.parametrize("T,Dk,Dv,decay", [(1, 64, 32, 2.0), (40, 64, 20, 2.0), (64, 128, 128, 0.2), (130, 64, 128, 0.2),
                                           (257, 128, 72, 2.0), (320, 64, 33, 0.2)])
def test_gated_delta_chunk_kernels(T, Dk, Dv, decay):
    """Gradients of fp32 inputs against the fp64 recurrence: fp32 sums, rounded once per product (the chunked PyTorch form is
    off by 1 to 3e-6 on the same inputs). The output is bf16."""
    from slowrun_b200.ops.linear_attention import gated_delta_rule
    B, H = 2, 3
    g = torch.Generator(device="cuda").manual_seed(T + Dv)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    norm = torch.nn.functional.normalize
    ins = [(norm(r(B, T, H, Dk), dim=-1) * Dk ** -0.5).bfloat16().float(), norm(r(B, T, H, Dk) + 0.5, dim=-1).bfloat16().float(),
           r(B, T, H, Dv).bfloat16().float(), -decay * torch.rand(B, T, H, device="cuda", generator=g),
           2 * torch.rand(B, T, H, device="cuda", generator=g)]
    w = r(B, T, H, Dv)
    a = [t.clone().requires_grad_() for t in ins]
    o = gated_delta_rule(*a)
    grads = torch.autograd.grad(o, a, w)
    q, k, v, gg, beta = (t.double().requires_grad_() for t in ins)
    S, out, d = torch.zeros(B, H, Dk, Dv, dtype=torch.float64, device="cuda"), [], torch.exp(gg)
    for t in range(T):
        S = S * d[:, t][..., None, None]
        S = S + beta[:, t][..., None, None] * k[:, t].unsqueeze(-1) * (v[:, t] - torch.einsum("bhkv,bhk->bhv", S, k[:, t])).unsqueeze(-2)
        out.append(torch.einsum("bhkv,bhk->bhv", S, q[:, t]))
    ref = torch.stack(out, 1)
    refs = torch.autograd.grad(ref, (q, k, v, gg, beta), w.double())
    _status_ok()
    assert _rel(o, ref.detach()) < 4e-3
    for x, y in zip(grads, refs):
        assert (x.double() - y).norm().item() < 2e-5 * y.norm().item() + 1e-12
