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


# --------------------------------------------------------------------------------------------- logits and distillation
@pytest.mark.parametrize("M,V,T,smoothing", [(1, 7, 0.5, 0.0), (5, 33, 1.0, 0.2), (64, 1000, 3.0, 0.0), (7, 50257, 1.0, 0.1)])
def test_distillation_terms(M, V, T, smoothing):
    """fp32 kernels against fp64: exponentials good to 2e-7 in sums of V terms."""
    import torch.nn.functional as F
    from slowrun_b200.ops import functional as ops
    g = torch.Generator(device="cuda").manual_seed(V)
    s, t = (3 * torch.randn(M, V, device="cuda", generator=g) for _ in range(2))
    y = torch.randint(0, V, (M,), device="cuda", generator=g)
    if M > 3:
        y[1] = -1
    a, b = s.clone().requires_grad_(), s.double().requires_grad_()
    ce, kl = ops.distill_terms(a, t, y, T, smoothing)
    grad, = torch.autograd.grad(0.3 * ce + 0.7 * kl, a)
    keep = y != -1
    ce64 = F.cross_entropy(b, y, label_smoothing=smoothing, ignore_index=-1)
    kl64 = F.kl_div(F.log_softmax(b[keep] / T, -1), F.log_softmax(t.double()[keep] / T, -1), reduction="batchmean", log_target=True)
    want, = torch.autograd.grad(0.3 * ce64 + 0.7 * kl64, b)
    assert _rel(ce.detach(), ce64.detach()) < 2e-6 and _rel(kl.detach(), kl64.detach()) < 4e-6 and _rel(grad, want) < 4e-6


@pytest.mark.parametrize("cap,vocab", [(15.0, 1001), (0.0, 1001), (10.0, 1008)])
def test_softcapped_logits(cap, vocab):
    from slowrun_b200.ops import functional as ops
    g = torch.Generator(device="cuda").manual_seed(vocab)
    x = (8 * torch.randn(3, 5, 1008, device="cuda", generator=g)).bfloat16()
    x[0, 0, :4] = torch.tensor([0.0, 1e-3, 300.0, -300.0])
    a, b = x.clone().requires_grad_(), x.double().requires_grad_()
    z, zr = ops._softcap_logits(a, cap, vocab), b[..., :vocab]
    zr = cap * torch.tanh(zr / cap) if cap > 0 else zr
    w = torch.randn(z.shape, device="cuda", generator=g)
    grad, = torch.autograd.grad(z, a, w)
    want, = torch.autograd.grad(zr, b, w.double())
    assert z.is_contiguous() and z.dtype == torch.float32
    assert _rel(z.detach(), zr.detach()) < 3e-7 and _rel(grad, want) < 4e-3          # fp32; bf16 gradient


# --------------------------------------------------------------------------------------------- block in one host call
@pytest.mark.parametrize("track,T", [("limited", 200), ("two_hour", 256), ("tiny", 328)])
def test_block_in_one_host_call_equals_the_calls_one_by_one(track, T, monkeypatch):
    """Same launches in the same order: losses agree to the bit, gradients up to the order of split-K and dQ additions, which
    differs between two runs of either path."""
    from slowrun_b200.config import track_defaults
    from slowrun_b200.models.gpt import build_model
    from slowrun_b200.ops import block as block_ops, functional as ops
    cfg = track_defaults(track)
    m = cfg.model
    m.n_layer, m.n_embd, m.n_head, m.n_kv_head, m.sequence_len = 4, 384, 3, 3, T
    model = build_model(m, torch.device("cuda"), seed=0)
    with torch.no_grad():
        for p in model.parameters():
            if not bool((p != 0).any()):
                p.normal_(0.0, 0.02)
    model.arena.refresh_shadows()
    idx = torch.randint(0, 50257, (2, T + 1), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    results = []
    for one_call in (True, False):
        if not one_call:
            monkeypatch.setattr(block_ops, "_one_call", lambda *a: False)
        torch.manual_seed(3)
        ops.set_dropout_rng_state({"salt": 0, "state": {("cuda", torch.cuda.current_device()): 5}})
        model.zero_grad_arena()
        out = model(idx[:, :-1], idx[:, 1:])
        loss = out[0] if isinstance(out, tuple) else out
        loss.backward()
        _status_ok()
        a = model.arena
        results.append((loss.item(), [t.clone() for t in [g.G for g in a.groups.values()] + [a.head_grad, a.small_grads]]))
    assert results[0][0] == results[1][0]
    for x, y in zip(*(r[1] for r in results)):
        assert (x - y).norm().item() <= 2e-2 * y.norm().item() + 1e-9
