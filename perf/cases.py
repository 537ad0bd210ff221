"""Performance cases of this framework on one GPU.

Every case goes through a public entry point: the fused model operators
(``flagcx_b200.ops``), a decoder block (``flagcx_b200.models.llama``), the tensor-core GEMM
(``flagcx_b200.parallel.tp``) and, as an emulated world of eight ranks on one GPU, the
collectives (``flagcx_b200.capi``) and the expert-parallel layer (``flagcx_b200.parallel.moe``).
"""
from __future__ import annotations

import functools
import weakref

import torch

from flagcx_b200 import capi, ops
from flagcx_b200.models.llama import LlamaConfig, build_units
from flagcx_b200.parallel.moe import MoeDispatcher, route
from flagcx_b200.parallel.tp import gemm_bf16

BF16 = torch.bfloat16
DTYPES = {"bf16": (torch.bfloat16, capi.BFLOAT16, 2), "fp16": (torch.float16, capi.HALF, 2),
          "fp32": (torch.float32, capi.FLOAT, 4)}
THETA, EPS = 500000.0, 1e-5
ADAM = dict(lr=3e-4, beta1=0.9, beta2=0.95, eps=1e-8, wd=0.1, step=10)


# ---- the cases ------------------------------------------------------------------------
def listed():
    return [
        # the pre-norm of a residual block, forward and backward: a training step's 4096 tokens
        # of the Llama-3-8B shape, and a short prompt on the tiny configuration, where what
        # counts is the latency of the call
        {"name": "norm_train", "kind": "norm", "rows": 4096, "hidden": 4096},
        {"name": "norm_short", "kind": "norm", "rows": 257, "hidden": 256},
        # rotary embedding over the fused projection, forward and backward, two sequences' worth
        {"name": "rope_train", "kind": "rope", "rows": 8192, "heads": 32, "kv_heads": 8, "head_dim": 128},
        # gated activation of the feed-forward part, forward and backward, an odd token count
        {"name": "swiglu_train", "kind": "swiglu", "rows": 4099, "ffn": 14336},
        # loss and gradient over the full vocabulary: the head of a training step
        {"name": "loss_train", "kind": "loss", "rows": 4096, "vocab": 128256},
        # optimizer step over the parameters of one Llama-3-8B layer
        {"name": "optimizer_layer", "kind": "adamw", "n": 218_112_000},
        # one tensor-parallel rank's column-parallel product: long prompts, and the fewest rows
        # that the kernel takes (decoding: the weights are streamed once)
        {"name": "gemm_prefill", "kind": "gemm", "m": 8192, "n": 3584, "k": 8192},
        {"name": "gemm_decode", "kind": "gemm", "m": 128, "n": 3584, "k": 8192},
        # all-reduce of eight ranks: one token's hidden state, and a gradient bucket with an odd count
        {"name": "allreduce_token", "kind": "allreduce", "count": 8192, "dtype": "bf16"},
        {"name": "allreduce_bucket", "kind": "allreduce", "count": (16 << 20) + 3, "dtype": "bf16"},
        # expert-parallel layer: 512 tokens a rank to their top 8 of 256 experts and back
        {"name": "moe_prefill", "kind": "moe", "tokens": 512, "hidden": 7168, "topk": 8, "experts": 256},
        # one whole decoder block, forward and backward, an odd sequence length
        {"name": "block_train", "kind": "block", "rows": 1021},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["norm", "rope", "swiglu", "loss", "adamw", "gemm", "gemm", "allreduce", "moe", "block"])
    if kind == "norm":
        return {"kind": kind, "rows": _log(rng, 1, 8192), "hidden": 8 * _log(rng, 32, 1024)}
    if kind == "rope":
        kv = rng.choice([1, 2, 4, 8])
        return {"kind": kind, "rows": _log(rng, 1, 8192), "heads": kv * rng.choice([1, 2, 4]), "kv_heads": kv,
                "head_dim": rng.choice([32, 64, 80, 96, 128])}
    if kind == "swiglu":
        return {"kind": kind, "rows": _log(rng, 1, 4096), "ffn": 8 * _log(rng, 64, 1792)}
    if kind == "loss":
        return {"kind": kind, "rows": _log(rng, 16, 4096), "vocab": 8 * _log(rng, 128, 16032)}
    if kind == "adamw":
        return {"kind": kind, "n": _log(rng, 1 << 10, 200_000_000)}
    if kind == "gemm":
        return {"kind": kind, "m": 128 * _log(rng, 1, 48), "n": 256 * _log(rng, 1, 24), "k": 64 * _log(rng, 4, 128)}
    if kind == "allreduce":
        return {"kind": kind, "count": _log(rng, 1 << 9, 12 << 20), "dtype": rng.choice(sorted(DTYPES))}
    if kind == "moe":
        return {"kind": kind, "tokens": _log(rng, 8, 400), "hidden": 128 * rng.randint(8, 56),
                "topk": rng.choice([2, 4, 6, 8]), "experts": rng.choice([64, 128, 256])}
    return {"kind": kind, "rows": _log(rng, 128, 1000)}


RANKS = 8


@functools.lru_cache(maxsize=1)
def _world():
    """One communicator per rank, kept as long as the program runs."""
    return capi.Comm.emu_world(RANKS, torch.cuda.current_device())


# ---- inputs -----------------------------------------------------------------------------
def _inputs(case, seed):
    """The tensors of a case, from the seed alone."""
    g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape, std=1.0, dtype=BF16):
        t = torch.empty(*shape, dtype=dtype, device="cuda")
        return t.normal_(0.0, std, generator=g)

    kind = case["kind"]
    if kind == "norm":
        r, h = case["rows"], case["hidden"]
        return {"x": normal(r, h), "w": 1 + normal(h, std=0.1), "g": normal(r, h), "g_skip": normal(r, h)}
    if kind == "rope":
        width = (case["heads"] + 2 * case["kv_heads"]) * case["head_dim"]
        return {"x": normal(case["rows"], width), "g": normal(case["rows"], width)}
    if kind == "swiglu":
        return {"x": normal(case["rows"], 2 * case["ffn"]), "g": normal(case["rows"], case["ffn"])}
    if kind == "loss":
        return {"logits": normal(case["rows"], case["vocab"], std=2.0),
                "targets": torch.randint(0, case["vocab"], (case["rows"],), generator=g, device="cuda")}
    if kind == "adamw":
        n = case["n"]
        return {"p": normal(n, std=0.02), "g": normal(n, std=1e-2), "m": normal(n, std=1e-3),
                "v": normal(n, std=1e-3).square_().add_(1e-6)}
    if kind == "gemm":
        return {"a": normal(case["m"], case["k"]), "b": normal(case["n"], case["k"], std=0.02)}
    if kind == "allreduce":
        return {"x": [normal(case["count"], dtype=DTYPES[case["dtype"]][0]) for _ in range(RANKS)]}
    if kind == "moe":
        t, h = case["tokens"], case["hidden"]
        x, idx, w = [], [], []
        for _ in range(RANKS):
            i, wt = route(normal(t, case["experts"], dtype=torch.float32), case["topk"])
            x.append(normal(t, h))
            idx.append(i)
            w.append(wt)
        return {"x": x, "idx": idx, "w": w}
    cfg = LlamaConfig.llama3_8b()
    unit = build_units(cfg)[1]
    params = [1 + normal(*s, std=0.1) if "norm" in name else normal(*s, std=cfg.init_std) for name, s in unit.shapes]
    return {"params": params, "x": normal(case["rows"], cfg.hidden), "g": normal(case["rows"], cfg.hidden)}


def _capacity(case):
    """Rows that a rank may receive: a quarter above the mean, and room for small batches."""
    return case["tokens"] * case["topk"] * 5 // 4 + 64 * case["topk"]


def _close(moes):
    for m in moes:
        m.close()


class _Layer:
    """The ranks' dispatchers of one expert-parallel layer."""

    def __init__(self, tokens, hidden, topk, experts, capacity):
        self.ranks = [MoeDispatcher(c, tokens, hidden, topk, experts, capacity) for c in _world()]
        weakref.finalize(self, _close, self.ranks)


# A program creates a layer once and keeps it; a pass uses it from dispatch to combine.
_layer = functools.lru_cache(maxsize=2)(_Layer)


def prepare(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    s["case"] = dict(case)
    if kind == "norm":
        for k in ("x", "w"):
            s[k].requires_grad_(True)
    elif kind in ("rope", "swiglu"):
        s["x"].requires_grad_(True)
    elif kind == "gemm":
        s["out"] = torch.empty(case["m"], case["n"], dtype=BF16, device="cuda")
    elif kind == "allreduce":
        _world()
        s["out"] = [torch.empty_like(t) for t in s["x"]]
    elif kind == "moe":
        s["layer"] = _layer(case["tokens"], case["hidden"], case["topk"], case["experts"], _capacity(case))
        s["out"] = [torch.empty_like(t) for t in s["x"]]
    elif kind == "block":
        s["fn"] = build_units(LlamaConfig.llama3_8b())[1].fn
        for t in s["params"] + [s["x"]]:
            t.requires_grad_(True)
    return s


# ---- one pass -----------------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "norm":
        y, skip = ops.rmsnorm_branch(s["x"], s["w"], EPS)
        dx, dw = torch.autograd.grad((y, skip), (s["x"], s["w"]), (s["g"], s["g_skip"]))
        return {"y": y, "dx": dx, "dw": dw}
    if kind == "rope":
        y = ops.rope_fused_qkv(s["x"], case["heads"], case["kv_heads"], case["head_dim"], THETA)
        (dx,) = torch.autograd.grad(y, s["x"], s["g"])
        return {"y": y, "dx": dx}
    if kind == "swiglu":
        y = ops.swiglu(s["x"])
        (dx,) = torch.autograd.grad(y, s["x"], s["g"])
        return {"y": y, "dx": dx}
    if kind == "loss":
        # the call turns the logits into their gradient; a second pass finds that gradient there
        # (in a program the head's GEMM writes new logits), which costs the same
        loss = ops.cross_entropy_(s["logits"], s["targets"])
        return {"loss": loss, "dlogits": s["logits"]}
    if kind == "adamw":
        a = ADAM
        ops.adamw_flat_(s["p"], s["g"], s["m"], s["v"], a["lr"], a["beta1"], a["beta2"], a["eps"], a["wd"], a["step"])
        return {"p": s["p"], "m": s["m"], "v": s["v"]}
    if kind == "gemm":
        return gemm_bf16(s["a"], s["b"], s["out"])
    if kind == "allreduce":
        dt = DTYPES[case["dtype"]][1]
        for comm, x, out in zip(_world(), s["x"], s["out"]):
            comm.all_reduce(x, out, case["count"], dt, capi.SUM)
        return s["out"]
    if kind == "moe":
        ranks = s["layer"].ranks
        for m, x, idx in zip(ranks, s["x"], s["idx"]):
            m.dispatch(x, idx)
        for m in ranks:  # where a program runs its experts: here they hand their rows back
            m.expert_out.copy_(m.recv_rows)
        for m, w, out in zip(ranks, s["w"], s["out"]):
            m.combine(w, out)
        return {"out": s["out"], "offsets": [m.expert_offsets for m in ranks]}
    y = s["fn"](s["params"], s["x"])
    grads = torch.autograd.grad(y, [s["x"]] + s["params"], s["g"])
    return {"y": y, "dx": grads[0], "dparams": list(grads[1:])}


# ---- what a pass cannot do without --------------------------------------------------------
def _block_params():
    return [s for _, s in build_units(LlamaConfig.llama3_8b())[1].shapes]


def work(case):
    kind = case["kind"]
    if kind == "norm":  # forward x -> y; backward g, g_skip, x -> dx
        n = case["rows"] * case["hidden"]
        return {"bytes": 2 * (6 * n + 2 * case["hidden"]), "flops": 16 * n}
    if kind == "rope":
        n = case["rows"] * (case["heads"] + 2 * case["kv_heads"]) * case["head_dim"]
        return {"bytes": 2 * 4 * n, "flops": 6 * n}
    if kind == "swiglu":  # forward ab -> y; backward ab, g -> dab
        n = case["rows"] * case["ffn"]
        return {"bytes": 2 * 8 * n, "flops": 20 * n}
    if kind == "loss":
        n = case["rows"] * case["vocab"]
        return {"bytes": 2 * 2 * n + 12 * case["rows"], "flops": 5 * n}
    if kind == "adamw":
        return {"bytes": 2 * 7 * case["n"], "flops": 15 * case["n"]}
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 2 * (m * k + n * k + m * n), "flops": 2 * m * n * k}
    if kind == "allreduce":
        size = DTYPES[case["dtype"]][2]
        return {"bytes": 2 * RANKS * case["count"] * size, "flops": (RANKS - 1) * case["count"]}
    if kind == "moe":  # tokens in, expert rows written, read and handed back, tokens out
        tokens, k = RANKS * case["tokens"], case["topk"]
        return {"bytes": 2 * case["hidden"] * tokens * (2 + 4 * k), "flops": 2 * case["hidden"] * tokens * k}
    t, cfg = case["rows"], LlamaConfig.llama3_8b()
    mats = sum(s[0] * s[1] for s in _block_params() if len(s) == 2)
    # weights read in each direction and their gradients written; activations between the parts
    return {"bytes": 2 * (3 * mats + t * (8 * cfg.hidden + 16 * cfg.ffn)),
            "flops": 6 * mats * t + 7 * t * t * cfg.hidden}


def tolerance(case):
    kind = case["kind"]
    if kind == "allreduce" and case["dtype"] == "fp32":
        return {"rel": 1e-6, "max": 1e-5}
    if kind == "allreduce" and case["dtype"] == "fp16":
        return {"rel": 1e-3, "max": 1e-2}
    if kind == "block":
        return {"rel": 2e-2, "max": 0.3}
    # one or two roundings to bf16 (2^-9 each, relative); "max": two units in the last place
    return {"rel": 6e-3, "max": 4e-2}


# ---- the same in 64 bits --------------------------------------------------------------------
def _rms64(x, w):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * w


def _rope64(x, rows, heads, head_dim, theta):
    """x: [rows, heads, head_dim], halves rotated against each other."""
    half = head_dim // 2
    inv = theta ** (-torch.arange(half, device=x.device, dtype=torch.float64) * 2 / head_dim)
    ang = torch.arange(rows, device=x.device, dtype=torch.float64)[:, None] * inv
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _rope_qkv64(x, case):
    d, rot = case["head_dim"], case["heads"] + case["kv_heads"]
    rows = x.shape[0]
    x = x.view(rows, -1, d)
    return torch.cat([_rope64(x[:, :rot], rows, rot, d, THETA), x[:, rot:]], 1).reshape(rows, -1)


def _swiglu64(x):
    a, b = x.chunk(2, -1)
    return torch.nn.functional.silu(a) * b


def _block64(params, x):
    cfg = LlamaConfig.llama3_8b()
    attn_norm, wqkv, wo, ffn_norm, w13, w2 = params
    t, nh, nkv, hd = x.shape[0], cfg.n_heads, cfg.n_kv_heads, cfg.head_dim
    q, k, v = (_rms64(x, attn_norm) @ wqkv.T).split([nh * hd, nkv * hd, nkv * hd], -1)
    q = _rope64(q.reshape(t, nh, hd), t, nh, hd, cfg.rope_theta)
    k = _rope64(k.reshape(t, nkv, hd), t, nkv, hd, cfg.rope_theta).repeat_interleave(nh // nkv, 1)
    v = v.reshape(t, nkv, hd).repeat_interleave(nh // nkv, 1)
    att = torch.einsum("qhd,khd->hqk", q, k) / hd ** 0.5
    att = att.masked_fill(torch.ones(t, t, device=x.device).triu(1).bool(), float("-inf")).softmax(-1)
    x = x + torch.einsum("hqk,khd->qhd", att, v).reshape(t, nh * hd) @ wo.T
    return x + _swiglu64(_rms64(x, ffn_norm) @ w13.T) @ w2.T


def exact(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    if kind in ("norm", "rope", "swiglu"):
        x = s["x"].double().requires_grad_(True)
        if kind == "norm":
            w = s["w"].double().requires_grad_(True)
            y = _rms64(x, w)
            dx, dw = torch.autograd.grad(y, (x, w), s["g"].double())
            return {"y": y.detach(), "dx": dx + s["g_skip"].double(), "dw": dw}
        y = _rope_qkv64(x, case) if kind == "rope" else _swiglu64(x)
        (dx,) = torch.autograd.grad(y, x, s["g"].double())
        return {"y": y.detach(), "dx": dx}
    if kind == "loss":
        logp = s["logits"].double().log_softmax(-1)
        at = torch.arange(case["rows"], device="cuda")
        loss = -logp[at, s["targets"]].mean()
        d = logp.exp_()
        d[at, s["targets"]] -= 1
        return {"loss": loss, "dlogits": d / case["rows"]}
    if kind == "adamw":
        a, g = ADAM, s["g"].double()
        m = a["beta1"] * s["m"].double() + (1 - a["beta1"]) * g
        v = a["beta2"] * s["v"].double() + (1 - a["beta2"]) * g * g
        upd = (m / (1 - a["beta1"] ** a["step"])) / ((v / (1 - a["beta2"] ** a["step"])).sqrt() + a["eps"])
        return {"p": s["p"].double() * (1 - a["lr"] * a["wd"]) - a["lr"] * upd, "m": m, "v": v}
    if kind == "gemm":
        return s["a"].double() @ s["b"].double().T
    if kind == "allreduce":
        total = sum(x.double() for x in s["x"])
        return [total] * RANKS
    if kind == "moe":
        per = case["experts"] // RANKS
        counts = sum(torch.bincount(i.flatten().long(), minlength=case["experts"]) for i in s["idx"]).view(RANKS, per)
        offsets = torch.nn.functional.pad(counts.cumsum(1), (1, 0))
        return {"out": [x.double() * w.double().sum(1, keepdim=True) for x, w in zip(s["x"], s["w"])],
                "offsets": list(offsets)}
    params = [p.double().requires_grad_(True) for p in s["params"]]
    x = s["x"].double().requires_grad_(True)
    y = _block64(params, x)
    grads = torch.autograd.grad(y, [x] + params, s["g"].double())
    return {"y": y.detach(), "dx": grads[0], "dparams": list(grads[1:])}
