"""The work that users of this framework have it do, as a list of measurable cases.

Every case goes through the calls a training or evaluation program makes: `build_model` and a forward/backward pass of one
micro-batch (all tracks), the per-token losses of an evaluation, the logits of a prompt, `ShardedMuonAdamW.step()`, and
`Trainer.train_step()` with its loader, CUDA graphs and optimizer. Sizes are those of the track defaults
(`slowrun_b200/config.py`), of `bench.py`, of the loss-parity runs and of the tests, or lie between them. Parameters that are
initialised to zero get small random values and the head trained-like magnitudes, so that every product of the network sees
the numbers it sees in the middle of a run and not those of its very first step.
"""
import gc
import os
import random
import shutil
import tempfile

import torch

from slowrun_b200.config import track_defaults
from slowrun_b200.data.synthetic import write_synthetic_corpus
from slowrun_b200.models.gpt import build_model
from slowrun_b200.models.hybrid import HybridGPT, HybridSpec, auto_linear_layers
from slowrun_b200.ops import functional as ops
from slowrun_b200.optim.groups import build_param_groups
from slowrun_b200.optim.muon_adamw import ShardedMuonAdamW
from slowrun_b200.parallel.comm import TorchComm
from slowrun_b200.train.trainer import Trainer
from slowrun_b200.train.unlimited import distillation_loss

DEVICE = "cuda"
HEAD_DIM = 128
HBM_BYTES_LIMIT = 50e9          # weights, gradients, activations of one drawn training case


def _case(name, kind, track, layers, heads, batch, seq, **more):
    return dict({"name": name, "kind": kind, "track": track, "layers": layers, "heads": heads, "batch": batch, "seq": seq}, **more)


def listed():
    return [
        # the smallest call: the smoke test's model, one micro-batch; latency and launch count
        _case("train_smoke", "train", "limited", 4, 2, 2, 256),
        # a research-sized model on ragged batches (no dimension of the token matrix is a multiple of a tile)
        _case("train_ragged", "train", "limited", 6, 5, 3, 1000),
        # the headline workload: one micro-batch of the 2.7B limited-track model
        _case("train_2.7b", "train", "limited", 30, 20, 4, 2048),
        # the two-hour track's default model in its middle window stage (YaRN) with replayed decoder layers
        _case("train_two_hour", "train", "two_hour", 30, 14, 4, 2048, short=768, long=1792, dupe=True),
        # the tiny track's default model at its default device batch: recurrence, XSA, fp8 head, multi-token loss
        _case("train_tiny", "train", "tiny", 16, 8, 32, 2048),
        # the unlimited track's chain distillation: student forward/backward and teacher forward on full logits
        _case("train_distill", "distill", "unlimited", 12, 16, 2, 2048),
        # the hybrid fork: Gated DeltaNet layers between softmax layers
        _case("train_hybrid", "hybrid", "limited", 4, 14, 4, 2048, square=False),
        # evaluation of the limited track's default model: per-token losses, no gradients
        _case("eval_1.4b", "eval", "limited", 30, 14, 4, 2048),
        # logits of one prompt of odd length
        _case("logits_prompt", "logits", "tiny", 16, 8, 1, 777),
        # one optimizer step on a slice of the 2.7B model's matrices (all its shapes)
        _case("optim_2.7b", "optim", "limited", 6, 20, 1, 2048),
        # one optimizer step of a small model: many small groups, launch-bound
        _case("optim_small", "optim", "limited", 8, 4, 1, 2048),
        # a whole training step through the Trainer: loader, CUDA-graph micro-batches, optimizer, loss read back
        _case("step_512", "step", "limited", 8, 4, 4, 2048, accum=2),
    ]


def draw(rng: random.Random):
    def log_int(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    while True:
        kind = rng.choice(["train", "train", "train", "train", "eval", "eval", "logits", "optim", "step", "distill", "hybrid"])
        track = rng.choice(["limited", "limited", "two_hour", "tiny"]) if kind in ("train", "eval", "logits") else \
            ("unlimited" if kind == "distill" else "limited")
        heads = rng.choice([2, 3, 4, 5, 6, 8, 10, 12, 14, 16, 20])
        layers = log_int(4, 16 if track == "tiny" else 30)
        seq = rng.choice([2048, 2048, 1024, log_int(100, 2048), log_int(100, 2048)])
        batch = log_int(1, 32 if track == "tiny" else 8)
        c = {"kind": kind, "track": track, "layers": layers, "heads": heads, "batch": batch, "seq": seq}
        if kind == "train" and track == "two_hour":
            c["long"] = max(2, int(seq * rng.choice([0.375, 0.625, 0.875])))
            c["short"] = max(1, int(c["long"] * rng.choice([0.33, 0.43, 0.625])))
            c["dupe"] = layers >= 8 and rng.random() < 0.5
        if kind == "hybrid":
            c["square"] = rng.random() < 0.5
            c["layers"], c["batch"] = min(layers, 6), min(batch, 4)
        if kind == "distill":
            c["layers"], c["batch"] = min(layers, 12), min(batch, 2)
        if kind == "logits":
            c["batch"] = min(batch, 2)
        if kind == "optim":
            c["layers"], c["batch"], c["seq"] = min(layers, 8), 1, 2048
        if kind == "step":
            c["layers"], c["heads"], c["seq"] = min(layers, 8), min(heads, 8), 2048
            c["batch"], c["accum"] = min(batch, 8), rng.choice([1, 2, 4])
        d = heads * HEAD_DIM
        activations = c["layers"] * c["batch"] * c["seq"] * d * 50
        if activations + 10 * _matrix_params(c) < HBM_BYTES_LIMIT and work(c)["flops"] <= work(listed()[2])["flops"]:
            return c


# ------------------------------------------------------------------------------------------------ sizes
def _hidden(d):
    return 256 * ((8 * d // 3 + 255) // 256)


def _matrix_params(c):
    """Parameters of the matrices that every token is multiplied with once (head and MTP block included)."""
    d = c["heads"] * HEAD_DIM
    per_layer = 4 * d * d + 3 * d * _hidden(d) + d * d / 2
    mtp = per_layer + 2 * d * d if c["track"] != "tiny" and c["kind"] != "hybrid" else 0
    return c["layers"] * per_layer + 50304 * d + mtp


def work(case):
    """Bytes: bf16 weights read, fp32 gradients (or updated state) written. Flops: the matrix products and the visible part
    of the attention products."""
    c = case
    d = c["heads"] * HEAD_DIM
    n, tokens = _matrix_params(c), c["batch"] * c["seq"]
    head = 50304 * d
    if c["kind"] == "optim":
        flops = 0
        for r, k, count in ((d, d, 4.5), (_hidden(d), d, 3)):           # five iterations of three products, two of them symmetric
            g, l = min(r, k), max(r, k)
            flops += 5 * (3 * g * g * l + g ** 3) * count * (c["layers"] + 1)
        return {"bytes": 26.0 * n + 34.0 * head, "flops": float(flops)}
    window_long = c.get("long", c["seq"])
    window_short = c.get("short", c["seq"] // 2)
    passes = c["layers"]
    if c.get("dupe"):
        lo, hi = _dupe_range(c)
        passes += 2 * (hi - lo)

    def pairs(w):
        w = min(w + 1, c["seq"])
        return w * c["seq"] - w * (w - 1) / 2

    mean_pairs = 0.75 * pairs(window_short) + 0.25 * pairs(window_long)
    attn_fwd = passes * 4.0 * mean_pairs * d * c["batch"]
    fwd = 2.0 * tokens * (n + (passes - c["layers"]) * (n - head) / (c["layers"] + 1)) + attn_fwd
    if c["kind"] in ("eval", "logits"):
        fwd *= 2 if c["track"] == "tiny" else 1
        out = tokens * 50257 * 4.0 if c["kind"] == "logits" else tokens * 4.0
        return {"bytes": 2.0 * n + out, "flops": fwd}
    train = 3.0 * fwd + 0.5 * attn_fwd                                   # backward of attention: five products for two
    nbytes = 2.0 * n + 4.0 * (n + head)
    if c["track"] == "tiny":
        train += fwd - 2.0 * tokens * head                               # the first pass of the recurrence has no backward
    if c["kind"] == "distill":
        train += fwd
        nbytes += 2.0 * n
    if c["kind"] == "step":
        o = work(dict(c, kind="optim"))
        return {"bytes": nbytes + o["bytes"], "flops": train * c["accum"] + o["flops"]}
    return {"bytes": nbytes, "flops": train}


def _dupe_range(c):
    """Replayed decoder layers: the limited track's 15..21 of 30, scaled to the depth."""
    lo = c["layers"] - c["layers"] // 2
    return lo, min(c["layers"], lo + max(1, c["layers"] // 5))


# ------------------------------------------------------------------------------------------------ inputs
def _config(c):
    cfg = track_defaults(c["track"])
    m = cfg.model
    m.n_layer, m.n_head, m.n_kv_head, m.n_embd, m.sequence_len = c["layers"], c["heads"], c["heads"], c["heads"] * HEAD_DIM, c["seq"]
    if c["kind"] == "hybrid":        # the fork's settings (research/hybrid_attn)
        m.stoch_depth, m.use_iha, m.iha_mix_v, m.mtp_weight, m.cproj_zero_init = 0.0, False, False, 0.0, True
    cfg.device_batch_size = c["batch"]
    return cfg


@torch.no_grad()
def _trained_like(model, gen):
    for p in model.parameters():
        if p.is_floating_point() and not bool((p != 0).any()):
            p.copy_(torch.randn(p.shape, device=p.device, generator=gen) * 0.02)
    model.lm_head.weight.normal_(0.0, 2.0 * model.config.n_embd ** -0.5, generator=gen)
    model.arena.refresh_shadows()


def _tokens(c, gen):
    """Token ids with their next-token targets, Zipf-Mandelbrot distributed like sub-word text (the most frequent id makes up
    one or two percent). The distribution function is summed on the host: a device scan rounds differently from run to run,
    and tokens would change with it."""
    w = 1.0 / (torch.arange(1, 50257, dtype=torch.float64) + 8.0)
    cdf = (w.cumsum(0) / w.sum()).to(DEVICE)
    u = torch.rand(c["batch"], c["seq"] + 1, device=DEVICE, dtype=torch.float64, generator=gen)
    rows = torch.searchsorted(cdf, u).clamp_(max=50255)
    return rows[:, :-1].contiguous(), rows[:, 1:].contiguous()


def _streams(seed):
    """The random streams of dropout and stochastic depth start from the seed."""
    torch.manual_seed(seed)
    ops.set_dropout_rng_state({"salt": 0, "state": {("cuda", torch.cuda.current_device()): seed}})


def _model(c, cfg, seed, gen):
    factory = None
    if c["kind"] == "hybrid":
        spec = HybridSpec(layers=auto_linear_layers(c["layers"]), head_dim_mode="square" if c["square"] else "param-matched")
        factory = lambda mc: HybridGPT(mc, spec)       # noqa: E731
    model = build_model(cfg.model, DEVICE, seed=seed, factory=factory)
    _trained_like(model, gen)
    if "long" in c:
        model.set_window_sizes(max(1, c["short"] // 2), max(1, c["long"] // 2))
        model.set_window_sizes(c["short"], c["long"], apply_yarn=True)
    if c.get("dupe"):
        model.set_dupe_layers(*_dupe_range(c), loops=2)
    return model.train(c["kind"] not in ("eval", "logits"))


class _TrainerState:
    """A Trainer on a synthetic corpus of its own; the corpus files go once the trainer has read them."""

    def __init__(self, c, cfg, seed, gen):
        folder = tempfile.mkdtemp(prefix="perf_corpus_")
        try:
            tokens = 8 * c["batch"] * c["accum"] * 2049 * 8
            write_synthetic_corpus(folder, train_tokens=tokens, val_tokens=20_000, seed=seed % 100_000)
            cfg.total_batch_size = c["batch"] * c["seq"] * c["accum"]
            cfg.input_bin, cfg.input_val_bin = (os.path.join(folder, f"fineweb_{n}.pt") for n in ("train", "val"))
            cfg.dupe_start_epoch = 10 ** 9
            self.trainer = Trainer(cfg, quiet=True)
        finally:
            shutil.rmtree(folder)
        _trained_like(self.trainer.model, gen)


def prepare(case, seed):
    gc.collect()          # models and their arenas refer to each other: an earlier state's memory only comes back here
    c, cfg = case, _config(case)
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    s = {"case": c}
    if c["kind"] == "step":
        s["trainer"] = _TrainerState(c, cfg, seed, gen).trainer
        _streams(seed)
        return s
    model = s["model"] = _model(c, cfg, seed, gen)
    if c["kind"] == "optim":
        s["optimizer"] = ShardedMuonAdamW(model, build_param_groups(model, cfg), TorchComm())
        a = model.arena
        for g in [g.G for g in a.groups.values()] + [a.head_grad, a.small_grads] + [p.grad for p in a.other_params]:
            g.normal_(0.0, 1e-3, generator=gen)
    else:
        s["x"], s["y"] = _tokens(c, gen)
        s["kw"] = {}
        if c["track"] == "tiny":
            s["kw"] = {"num_iterations": cfg.model.num_iterations}
            if c["kind"] == "train":
                s["kw"]["mtp_weights"] = torch.tensor([1.0, 0.5, 0.25], device=DEVICE)
    if c["kind"] == "distill":
        s["teacher"] = _model(c, cfg, seed + 1_000_003, gen).eval()
        s["cfg"] = cfg
    _streams(seed)
    return s


# ------------------------------------------------------------------------------------------------ passes
def _gradients(model):
    a = model.arena
    return [g.G for g in a.groups.values()] + [a.head_grad, a.small_grads] + [p.grad for p in a.other_params]


def _weights(model):
    a = model.arena
    return [g.P for g in a.groups.values()] + [model.lm_head.weight.data, a.small_P] + [p.data for p in a.other_params]


def run(state):
    s = state
    kind = s["case"]["kind"]
    if kind == "step":
        out = s["trainer"].train_step(sync=True)
        return {"loss": out["loss"], "weights": _weights(s["trainer"].model)}
    model = s["model"]
    if kind == "optim":
        opt = s["optimizer"]
        opt.step()
        momenta = [opt.state[g["name"]]["momentum"] for g in opt.param_groups if g["kind"] == "muon"]
        return {"weights": _weights(model), "momenta": momenta}
    if kind == "eval":
        with torch.no_grad():
            return model(s["x"], s["y"], loss_reduction="none", **s["kw"])
    if kind == "logits":
        with torch.no_grad():
            return model(s["x"], **s["kw"])
    model.zero_grad_arena()
    if kind == "distill":
        cfg = s["cfg"]
        logits, mtp_loss = model(s["x"], s["y"], distill=True)
        with torch.no_grad():
            teacher = s["teacher"](s["x"])
        loss = distillation_loss(logits, teacher, s["y"], mtp_loss, model.mtp_weight, cfg.distill_alpha, cfg.distill_temperature)
    else:
        out = model(s["x"], s["y"], **s["kw"])
        loss = out[0] if isinstance(out, tuple) else out
    loss.backward()
    return {"loss": loss.detach(), "gradients": _gradients(model)}


def tolerance(case):
    """Four times (and at most 3 %) what the same pass differs by when the blocks run operation by operation and the head as
    separate product and loss, which rounds the same bf16 intermediates at other places: 0.2 % on per-token losses, 1.2 % on
    logits, 1 % on gradients (0.5 % on the tiny track, 3 % on the short convolutions of the hybrid), 1.5 % on the head gates
    after an optimizer step. `max` is set by single rows of the embedding gradient, which are sums over few tokens."""
    kind = case["kind"]
    if kind == "eval":
        return {"rel": 0.008, "max": 0.03}
    if kind == "logits":
        return {"rel": 0.03, "max": 0.3}
    if kind == "optim":                 # Newton-Schulz in bf16 from norms summed in another order
        return {"rel": 0.003, "max": 0.1}
    if kind == "step":
        return {"rel": 0.03, "max": 0.4}
    return {"rel": 0.02 if case["track"] == "tiny" else 0.03, "max": 0.9}
