"""Workloads that time and check the framework's GPU path through its public entry points.

Each case is one layer or block of the hybrid models (delta-rule attention, softmax attention, the
SwiGLU FFN, the expert FFN, the normalisation, the vocabulary head) or one whole trainer step, at
the sizes that the repository's configurations, tests and benchmark use: ``listed()`` names a few,
``draw(rng)`` picks another one from the same ranges. ``prepare`` makes what a program has in hand
before the call, ``run`` is one call, ``exact`` the same result in 64-bit torch.
"""
from __future__ import annotations

import math

import torch

from prometheus_b200 import engine, kernels, model, train
from prometheus_b200.ops import attention, fp8, moe
from prometheus_b200.ops import functional as ops

BF16 = torch.bfloat16
CAP = 30.0          # soft cap of the logits


def listed() -> list:
    return [
        # one delta-rule layer of the 1.3B hybrid in training: 4 sequences of a micro-batch
        {"name": "delta_train", "kind": "delta", "batch": 4, "seq": 4096, "heads": 16, "grad": True, "state": False},
        # the same layer reading one long context (prefill / evaluation) with a state carried in
        {"name": "delta_long", "kind": "delta", "batch": 1, "seq": 16384, "heads": 16, "grad": False, "state": True},
        # a short odd-length fine-tuning batch on a small model: launches and latency
        {"name": "delta_short", "kind": "delta", "batch": 2, "seq": 200, "heads": 4, "grad": True, "state": False},
        # one grouped-query softmax layer of the 1.3B hybrid in training
        {"name": "attention_train", "kind": "attention", "batch": 4, "seq": 4096, "q_heads": 16, "kv_heads": 4,
         "grad": True, "max_logit": False},
        # evaluation of a ragged batch with the QK-clip statistic (largest logit per row)
        {"name": "attention_ragged", "kind": "attention", "batch": 3, "seq": 1000, "q_heads": 16, "kv_heads": 4,
         "grad": False, "max_logit": True},
        # the dense SwiGLU FFN of the 1.3B hybrid, four sequences of 4096 tokens, bf16
        {"name": "mlp_train", "kind": "mlp", "tokens": 16384, "d": 2048, "hidden": 5632, "fp8": False, "grad": True},
        # a shared expert of the 16B mixture (block-scaled FP8 linears), a ragged token count
        {"name": "mlp_fp8_train", "kind": "mlp", "tokens": 5000, "d": 2048, "hidden": 1408, "fp8": True, "grad": True},
        # one expert layer of the 16B mixture: 64 routed top-6 and 2 shared experts, FP8 products
        {"name": "moe_fp8_train", "kind": "moe", "tokens": 8192, "d": 2048, "hidden": 1408, "experts": 64,
         "shared": 2, "top_k": 6, "fp8": True, "grad": True},
        # the expert layer of the tiny reference model, evaluated on one sequence of 512 tokens
        {"name": "moe_small", "kind": "moe", "tokens": 512, "d": 256, "hidden": 512, "experts": 8, "shared": 0,
         "top_k": 2, "fp8": False, "grad": False},
        # residual add + RMSNorm of the 1.3B hybrid, forward and backward
        {"name": "norm_train", "kind": "norm", "rows": 16384, "d": 2048, "grad": True},
        # soft-capped cross-entropy over the 131072-word vocabulary with its gradients
        {"name": "head_train", "kind": "head", "rows": 4096, "d": 2048, "vocab": 131072, "grad": True},
        # one optimizer step (two micro-batches, Muon + AdamW) of a four-layer hybrid
        {"name": "step", "kind": "step", "batch": 4, "seq": 1024, "d": 1024, "layers": 4, "hidden": 2816,
         "vocab": 16384},
    ]


def _log(rng, lo: int, hi: int, mult: int = 1) -> int:
    return max(mult, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / mult)) * mult)


def draw(rng) -> dict:
    kind = rng.choice(["delta", "delta", "attention", "attention", "mlp", "mlp", "moe", "moe", "norm", "head"])
    grad = rng.random() < 0.6
    if kind == "delta":
        heads, seq = rng.choice([2, 4, 8, 16]), _log(rng, 64, 16384)
        batch = rng.randint(1, max(1, min(8, 16384 * 16 // (seq * heads))))
        return {"kind": kind, "batch": batch, "seq": seq, "heads": heads, "grad": grad, "state": rng.random() < 0.3}
    if kind == "attention":
        kv, seq = rng.choice([1, 2, 4]), _log(rng, 64, 8192)
        q_heads = kv * rng.choice([1, 2, 4])
        batch = rng.randint(1, max(1, min(8, 4 * 4096 * 4096 * 16 // (seq * seq * q_heads))))
        return {"kind": kind, "batch": batch, "seq": seq, "q_heads": q_heads, "kv_heads": kv, "grad": grad,
                "max_logit": rng.random() < 0.3}
    if kind == "mlp":
        return {"kind": kind, "tokens": _log(rng, 64, 16384), "d": rng.choice([512, 1024, 2048]),
                "hidden": 128 * rng.randint(4, 44), "fp8": rng.random() < 0.5, "grad": grad}
    if kind == "moe":
        experts = rng.choice([8, 16, 32, 64])
        return {"kind": kind, "tokens": _log(rng, 64, 8192), "d": rng.choice([256, 1024, 2048]),
                "hidden": 128 * rng.randint(4, 11), "experts": experts, "shared": rng.randint(0, 2),
                "top_k": rng.choice([2, 4, 6]), "fp8": rng.random() < 0.5, "grad": grad}
    if kind == "norm":
        return {"kind": kind, "rows": _log(rng, 64, 32768), "d": 128 * rng.randint(2, 16), "grad": grad}
    return {"kind": "head", "rows": _log(rng, 64, 6144), "d": rng.choice([512, 1024, 2048]),
            "vocab": _log(rng, 8192, 131072, 8), "grad": grad}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, *shape, scale: float = 1.0) -> torch.Tensor:
    x = torch.empty(shape, dtype=BF16, device="cuda").normal_(generator=g)
    return x.mul_(scale) if scale != 1.0 else x


def _unit(g, *shape) -> torch.Tensor:
    x = torch.empty(shape, dtype=torch.float32, device="cuda").normal_(generator=g)
    return torch.nn.functional.normalize(x, dim=-1).to(BF16)


def prepare(case: dict, seed: int) -> dict:
    g = _gen(seed)
    kind = case["kind"]
    s = {"case": case, "params": [], "gout": []}
    if kind == "delta":
        b, n, h = case["batch"], case["seq"], case["heads"]
        # unit keys and queries, write gates through a sigmoid, as the model feeds the layer
        s["params"] = [_unit(g, b, n, h, 128), _unit(g, b, n, h, 128), _randn(g, b, n, h, 128),
                       torch.sigmoid(_randn(g, b, n, h))]
        if case["state"]:
            s["state"] = torch.empty((b, h, 128, 128), device="cuda").normal_(generator=g) * 0.3
        s["gout"] = [_randn(g, b, n, h, 128)]
    elif kind == "attention":
        b, n, hq, hkv = case["batch"], case["seq"], case["q_heads"], case["kv_heads"]
        s["params"] = [_randn(g, b, n, hq, 128), _randn(g, b, n, hkv, 128), _randn(g, b, n, hkv, 128)]
        s["gout"] = [_randn(g, b, n, hq, 128)]
    elif kind == "mlp":
        t, d, h = case["tokens"], case["d"], case["hidden"]
        s["params"] = [_randn(g, t, d), _randn(g, 2 * h, d, scale=d ** -0.5), _randn(g, d, h, scale=h ** -0.5)]
        s["gout"] = [_randn(g, t, d)]
    elif kind == "moe":
        t, d, h, e = case["tokens"], case["d"], case["hidden"], case["experts"]
        n = e + case["shared"]
        s["params"] = [_randn(g, t, d), _randn(g, e, d, scale=d ** -0.5), _randn(g, n, 2 * h, d, scale=d ** -0.5),
                       _randn(g, n, d, h, scale=h ** -0.5)]
        # the balancing bias of a run that has been going for a while: far larger than the
        # rounding of a score, so that selections are the same for every correct arithmetic
        s["bias"] = torch.empty(e, device="cuda").normal_(generator=g) * 0.02
        s["gout"] = [_randn(g, t, d)]
    elif kind == "norm":
        r, d = case["rows"], case["d"]
        w = 1.0 + 0.1 * torch.empty(d, device="cuda").normal_(generator=g)
        s["params"] = [_randn(g, r, d), _randn(g, r, d), w]
        s["gout"] = [_randn(g, r, d), _randn(g, r, d)]
    elif kind == "head":
        r, d, v = case["rows"], case["d"], case["vocab"]
        s["params"] = [_randn(g, r, d), _randn(g, v, d, scale=0.02)]
        s["targets"] = torch.randint(0, v, (r,), generator=g, device="cuda", dtype=torch.int32)
        s["wt"] = torch.full((r,), 1.0 / r, device="cuda")
    else:
        cfg = model.ModelConfig(
            d_model=case["d"], n_layers=case["layers"], n_dense=case["layers"], n_moe=0,
            n_linear_attn=case["layers"] - case["layers"] // 4, n_mla=case["layers"] // 4, n_routed_experts=1,
            n_shared_experts=0, top_k=1, expert_hidden=512, mtp_heads=0, core_block_layers=case["layers"],
            recurrence_train_mean=1.0, recurrence_max=1, vocab_size=case["vocab"], max_context=case["seq"],
            prelude_layers=0, coda_layers=0, adapter_hidden=256, n_heads=case["d"] // 128, d_head=128,
            n_kv_heads=max(1, case["d"] // 512), softmax_kind="gqa", softmax_every=4, delta_beta="sigmoid", chunk=64,
            dense_hidden=case["hidden"])
        tcfg = train.train_config_for(cfg, warmup_steps=200, stable_steps=2000, decay_steps=200)
        s["trainer"] = engine.Trainer(cfg, tcfg, seed=seed, device="cuda", micro_batch=max(1, case["batch"] // 2))
        s["tokens"] = torch.randint(0, case["vocab"], (case["batch"], case["seq"]), generator=g, device="cuda")
        return s
    if case["grad"]:
        for p in s["params"]:
            p.requires_grad_(True)
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _ffn(x, w_gu, w_down, use_fp8: bool):
    f = fp8.fp8_linear if use_fp8 else ops.linear
    return f(ops.swiglu(f(x, w_gu)), w_down)


def run(s: dict):
    c = s["case"]
    kind = c["kind"]
    if kind == "step":
        tr = s["trainer"]
        out = tr.step(s["tokens"])
        return {"loss": out["loss"], "grad_norm": out["grad_norm"], "muon": tr.muon_master, "adam": tr.adam_master,
                "vec": tr.vec_master}
    with torch.set_grad_enabled(c["grad"]):
        p = s["params"]
        if kind == "delta":
            out, fin = kernels.chunked_delta_rule(p[0], p[1], p[2], p[3], s.get("state"))
            outs, extra = [out], [fin.detach()]
        elif kind == "attention":
            if c["max_logit"]:
                out, top = attention.causal_gqa(p[0], p[1], p[2], return_max_logit=True)
                outs, extra = [out], [top]
            else:
                outs, extra = [attention.causal_gqa(p[0], p[1], p[2])], []
        elif kind == "mlp":
            outs, extra = [_ffn(p[0], p[1], p[2], c["fp8"])], []
        elif kind == "moe":
            out, probs, ids = moe.moe_ffn(p[0], p[1], s["bias"], p[2], p[3], c["top_k"], n_shared=c["shared"],
                                          fp8=c["fp8"])
            outs, extra = [out], [probs.detach(), ids]
        elif kind == "norm":
            outs, extra = list(ops.add_rmsnorm(p[0], p[1], p[2])), []
        else:
            outs, extra = [ops.softcap_cross_entropy(p[0], p[1], s["targets"], s["wt"], CAP)], []
    grads = []
    if c["grad"]:
        grads = list(torch.autograd.grad(outs, p, s["gout"] if s["gout"] else None))
    return {"out": [o.detach() for o in outs], "extra": extra, "grads": grads}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case: dict) -> dict:
    kind = case["kind"]
    g = case.get("grad", True)
    if kind == "delta":
        b, n, h = case["batch"], case["seq"], case["heads"]
        tok = b * n * h
        # forward: read q, k, v, write out; backward: also read d(out), write dq, dk, dv
        byt = tok * 128 * 2 * (4 + (7 if g else 0)) + tok * 2 * (3 if g else 1)
        byt += b * h * 128 * 128 * 4 * (2 if case["state"] else 1)
        # per 64-token chunk: K K^T, the solve's two products, Q K^T, W S, Q S, M U, K^T U
        flops = tok / 64 * 2.0 * (4 * 64 * 64 * 128 + 3 * 64 * 128 * 128 + 64 * 64 * 128)
        return {"bytes": byt, "flops": flops * (3 if g else 1)}
    if kind == "attention":
        b, n, hq, hkv = case["batch"], case["seq"], case["q_heads"], case["kv_heads"]
        byt = b * n * 128 * 2 * (2 * hq + 2 * hkv) + (b * n * hq * 4 if case["max_logit"] else 0)
        flops = 2.0 * 2 * 128 * b * hq * n * (n + 1) / 2
        if g:
            byt += b * n * 128 * 2 * (3 * hq + 4 * hkv)
            flops *= 3.5
        return {"bytes": byt, "flops": flops}
    if kind == "mlp":
        t, d, h = case["tokens"], case["d"], case["hidden"]
        wt, x = 3 * d * h * 2, t * d * 2
        return {"bytes": (2 * x + wt) + ((2 * x + wt) if g else 0), "flops": 2.0 * t * 3 * d * h * (3 if g else 1)}
    if kind == "moe":
        t, d, h, e, sh, k = (case[x] for x in ("tokens", "d", "hidden", "experts", "shared", "top_k"))
        wt = ((e + sh) * 3 * d * h + e * d) * 2
        byt = 2 * t * d * 2 + wt + t * (4 * e + 4 * k)
        flops = 2.0 * t * (3 * d * h * (k + sh) + d * e)
        if g:
            byt += 2 * t * d * 2 + wt
            flops *= 3
        return {"bytes": byt, "flops": flops}
    if kind == "norm":
        n = case["rows"] * case["d"]
        return {"bytes": n * 2 * (4 + (4 if g else 0)) + 4 * case["d"] * (2 if g else 1),
                "flops": 4.0 * n + (8.0 * n if g else 0)}
    if kind == "head":
        r, d, v = case["rows"], case["d"], case["vocab"]
        return {"bytes": (r * d + v * d) * 2 * (2 if g else 1), "flops": 2.0 * r * d * v * (3 if g else 1)}
    t, d, L, v = case["batch"] * case["seq"], case["d"], case["layers"], case["vocab"]
    per = 3 * d * case["hidden"] + 4 * d * d
    mats = L * per
    # fp32 master, momentum, gradient read and written, bf16 copy written; five Newton-Schulz steps
    ns = L * 5 * 2.0 * (4 * (3 * d ** 3) + 3 * (2 * d * d * case["hidden"] + d ** 3))
    return {"bytes": mats * 22.0 + 2 * v * d * 30.0, "flops": 6.0 * t * (mats + v * d) + ns}


def tolerance(case: dict):
    """Each path was measured against ``exact``; two correct implementations at the same precision
    (bf16 operands and stored intermediates, fp32 sums) differ by up to that many parts each."""
    kind = case["kind"]
    if kind == "step":                       # masters after one update of a few parts in 10^4
        return {"rel": 5e-3, "max": 0.9}
    if kind == "norm":                       # 2e-3 off: one bf16 rounding
        return {"rel": 8e-3, "max": 0.05}
    if kind == "head":                       # 2e-3 off
        return {"rel": 8e-3, "max": 0.2}
    if kind == "moe" or case.get("fp8"):     # 2e-2 off: roundings before e4m3 move some values by a whole e4m3 step
        return {"rel": 3e-2, "max": 0.9, "differ": 2e-3}
    return {"rel": 1.5e-2, "max": 0.5}       # 4e-3 to 5e-3 off


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _delta64(q, k, v, beta, state):
    b, n, h, d = q.shape
    pad = (-n) % 64
    if pad:
        q, k, v = (torch.nn.functional.pad(t, (0, 0, 0, 0, 0, pad)) for t in (q, k, v))
        beta = torch.nn.functional.pad(beta, (0, 0, 0, pad))
    nc = (n + pad) // 64
    qc, kc, vc = (t.reshape(b, nc, 64, h, d).permute(0, 3, 1, 2, 4) for t in (q, k, v))
    bc = beta.reshape(b, nc, 64, h).permute(0, 3, 1, 2)
    eye = torch.eye(64, dtype=q.dtype, device=q.device)
    a = eye + torch.tril(bc[..., None] * (kc @ kc.transpose(-1, -2)), -1)
    rhs = torch.cat([bc[..., None] * kc, bc[..., None] * vc], dim=-1)
    sol = torch.linalg.solve_triangular(a, rhs, upper=False, unitriangular=True)
    w, uh = sol[..., :d], sol[..., d:]
    m = torch.tril(qc @ kc.transpose(-1, -2))
    st = torch.zeros((b, h, d, d), dtype=q.dtype, device=q.device) if state is None else state
    outs = []
    for i in range(nc):
        u = uh[:, :, i] - w[:, :, i] @ st
        outs.append(qc[:, :, i] @ st + m[:, :, i] @ u)
        st = st + kc[:, :, i].transpose(-1, -2) @ u
    out = torch.stack(outs, 2).permute(0, 2, 3, 1, 4).reshape(b, nc * 64, h, d)[:, :n]
    return out, st


def _attention64(q, k, v):
    b, n, hq, d = q.shape
    rep = hq // k.shape[2]
    mask = torch.ones(n, n, dtype=torch.bool, device=q.device).tril()
    rows, tops = [], []
    for i in range(b):
        heads = []
        for j in range(hq):
            lg = (q[i, :, j] @ k[i, :, j // rep].t()) / math.sqrt(d)
            lg = lg.masked_fill(~mask, float("-inf"))
            tops.append(lg.detach().amax(-1))
            heads.append(torch.softmax(lg, -1) @ v[i, :, j // rep])
        rows.append(torch.stack(heads, 1))
    return torch.stack(rows), torch.stack(tops).view(b, hq, n)


def _e4m3(x, scale):
    return (x.float() / scale).to(torch.float8_e4m3fn).double() * scale.double()


def _q_rows(x):
    """1 x 128 blocks, straight-through gradient."""
    xf = x.detach().float()
    t = xf.view(xf.shape[0], -1, 128)
    am = t.abs().amax(-1, keepdim=True)
    sc = torch.where(am > 0, am / 448.0, torch.ones_like(am))
    return x + (_e4m3(t, sc).view(xf.shape) - x.detach())


def _q_blocks(w):
    """128 x 128 blocks of a matrix, straight-through gradient."""
    wf = w.detach().float()
    n, k = wf.shape
    pad = (-n) % 128
    t = torch.nn.functional.pad(wf, (0, 0, 0, pad)).view(-1, 128, k // 128, 128)
    am = t.abs().amax(dim=(1, 3), keepdim=True)
    sc = torch.where(am > 0, am / 448.0, torch.ones_like(am))
    return w + (_e4m3(t, sc).view(n + pad, k)[:n] - w.detach())


def _ffn64(x, w_gu, w_down, use_fp8):
    h = w_down.shape[1]
    gu = _q_rows(x) @ _q_blocks(w_gu).t() if use_fp8 else x @ w_gu.t()
    hs = torch.nn.functional.silu(gu[:, :h]) * gu[:, h:]
    return _q_rows(hs) @ _q_blocks(w_down).t() if use_fp8 else hs @ w_down.t()


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "step":
        return None
    s = prepare(case, seed)
    p = [t.detach().double().requires_grad_(case["grad"]) for t in s["params"]]
    with torch.set_grad_enabled(case["grad"]):
        if kind == "delta":
            st = s["state"].double() if "state" in s else None
            out, fin = _delta64(*p, st)
            outs, extra = [out], [fin.detach()]
        elif kind == "attention":
            if case["grad"] and case["batch"] * case["q_heads"] * case["seq"] ** 2 > 1.2e9:
                return None          # the saved probabilities would not fit
            out, top = _attention64(*p)
            outs, extra = [out], [top] if case["max_logit"] else []
        elif kind == "mlp":
            outs, extra = [_ffn64(*p, case["fp8"])], []
        elif kind == "moe":
            x, rw, w_gu, w_down = p
            probs = torch.sigmoid(x @ rw.t())
            ids = torch.argsort(-(probs.detach() + s["bias"].double()), dim=-1, stable=True)[:, :case["top_k"]]
            top = torch.gather(probs, 1, ids)
            gates = top / top.sum(-1, keepdim=True).clamp_min(1e-9)
            out = torch.zeros_like(x)
            for e in range(case["experts"] + case["shared"]):
                if e < case["experts"]:
                    rows, slot = (ids == e).nonzero(as_tuple=True)
                    if rows.numel():
                        y = _ffn64(x[rows], w_gu[e], w_down[e], case["fp8"])
                        out = out.index_add(0, rows, gates[rows, slot, None] * y)
                else:
                    out = out + _ffn64(x, w_gu[e], w_down[e], case["fp8"])
            outs, extra = [out], [probs.detach(), None]
        elif kind == "norm":
            h = p[0] + p[1]
            outs, extra = [h * torch.rsqrt(h.square().mean(-1, keepdim=True) + 1e-6) * p[2], h], []
        else:
            total = 0.0
            for r0 in range(0, case["rows"], 1024):
                lg = CAP * torch.tanh(p[0][r0:r0 + 1024] @ p[1].t() / CAP)
                nll = torch.nn.functional.cross_entropy(lg, s["targets"][r0:r0 + 1024].long(), reduction="none")
                total = total + (nll * s["wt"][r0:r0 + 1024].double()).sum()
            outs, extra = [total], []
    grads = []
    if case["grad"]:
        go = [t.double() for t in s["gout"]] if s["gout"] else None
        grads = list(torch.autograd.grad(outs, p, go))
    return {"out": [o.detach() for o in outs], "extra": extra, "grads": grads}
