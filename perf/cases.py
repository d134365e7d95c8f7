"""The performance cases of this library: what a user of it runs, through its public entry points.

A case is a dict of plain values; ``kind`` names the entry points it goes through:

  model      StackedMAG.step_graphed: one whole training step (forward, backward, clip, AdamW)
  single     MAGSingle.loss_and_grads: the fp32 single-block configuration, eager
  exact      the exact memory-rule pair on stored trajectories (titans/delta_*_dd), forward + backward
  chunkwise  the frozen-M0 chunkwise pair (titans/delta_chunkwise_*_dd), forward + backward
  swa        sliding-window attention in bf16 (swa_forward_lse / swa_backward_lse)
  mlp        the Titans rule with a two-layer MLP memory (titans_mlp_*_dd), forward + backward
  adamw      FlatAdamW.step: global-norm clip and multi-tensor AdamW over one arena

Problems of the rule pairs are batch x heads independent memories; sizes that are not multiples of a
tile, a chunk or a power of two are part of the ranges.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from nl_hecate_b200 import dispatch as D
from nl_hecate_b200.mag_single import MAGSingle
from nl_hecate_b200.optimizer import FlatAdamW
from nl_hecate_b200.stacked_mag import StackedMAG, StackedMAGConfig


def listed():
    return [
        # the training step of the stacked model on one GPU at its full global batch
        {"name": "model_batch64", "kind": "model", "batch": 64, "seq": 512, "d_model": 512, "heads": 8, "blocks": 4},
        # the same step on one of eight data-parallel ranks: small kernels, bound by latency
        {"name": "model_batch8", "kind": "model", "batch": 8, "seq": 512, "d_model": 512, "heads": 8, "blocks": 4},
        # the smallest model: one block, one head, fp32, eager; what a first experiment or a test runs
        {"name": "single_delta_fp32", "kind": "single", "rule": "delta", "batch": 2, "seq": 256, "d_model": 64,
         "heads": 1, "window": 256, "vocab": 256},
        # the chunkwise kernel pair of a training step at long sequences: batch 16 x 8 heads
        {"name": "chunkwise_titans", "kind": "chunkwise", "rule": "titans", "problems": 128, "seq": 2048, "d": 64,
         "chunk": 64},
        # a ragged batch of the chunkwise Delta rule: no size is a multiple of the chunk
        {"name": "chunkwise_delta_ragged", "kind": "chunkwise", "rule": "delta", "problems": 24, "seq": 1000, "d": 64,
         "chunk": 48},
        # the drop-in exact pair with both trajectories stored, as a host of the C ABI calls it
        {"name": "exact_titans", "kind": "exact", "rule": "titans", "problems": 128, "seq": 2048, "d": 64,
         "store_s": True},
        # one sequence of eight heads through the exact rule: a latency-bound call
        {"name": "exact_titans_one_seq", "kind": "exact", "rule": "titans", "problems": 8, "seq": 333, "d": 64,
         "store_s": False},
        # heads of 128 through the exact Delta (DGD) rule
        {"name": "exact_delta_d128", "kind": "exact", "rule": "delta", "problems": 16, "seq": 512, "d": 128,
         "store_s": True},
        # attention of a training step at long context
        {"name": "swa_long", "kind": "swa", "batch": 8, "heads": 16, "seq": 8192, "hd": 64, "window": 512},
        # attention over a short sequence that fills no tile
        {"name": "swa_ragged", "kind": "swa", "batch": 2, "heads": 8, "seq": 777, "hd": 64, "window": 256},
        # deep (MLP) memory of the Titans rule over a training batch
        {"name": "mlp_titans", "kind": "mlp", "problems": 128, "seq": 256, "d": 64, "hidden": 256, "activation": 0},
        # the optimizer step over the stacked model's parameters
        {"name": "adamw_25m", "kind": "adamw", "params": 25_200_000, "tensors": 109},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("model", "single", "chunkwise", "chunkwise", "exact", "exact", "swa", "swa", "mlp", "adamw"))
    if kind == "model":
        # sequences are a multiple of every level's chunk: multiples of 64 up to 512, or 1024
        seq = rng.choice((128, 192, 256, 320, 448, 512, 512, 1024))
        heads = rng.choice((4, 8, 8))
        return {"kind": kind, "batch": _log(rng, 1, 32768 // max(seq, 512)), "seq": seq, "d_model": 64 * heads,
                "heads": heads, "blocks": rng.choice((2, 4, 4))}
    if kind == "single":
        heads, hd = rng.choice(((1, 64), (1, 32), (2, 32)))
        return {"kind": kind, "rule": rng.choice(("delta", "titans")), "batch": rng.randint(1, 8),
                "seq": _log(rng, 32, 512), "d_model": heads * hd, "heads": heads,
                "window": rng.choice((32, 64, 128, 256)), "vocab": rng.choice((128, 256, 512))}
    if kind == "chunkwise":
        seq = _log(rng, 48, 4096)
        return {"kind": kind, "rule": rng.choice(("titans", "titans", "delta")), "seq": seq,
                "problems": _log(rng, 4, min(512, 262144 // seq)), "d": rng.choice((64, 64, 64, 32)),
                "chunk": rng.choice((8, 16, 24, 32, 48, 64, 64))}
    if kind == "exact":
        d = rng.choice((64, 64, 64, 32, 128))
        seq = _log(rng, 24, 2048 if d < 128 else 512)
        rule = rng.choice(("titans", "titans", "delta"))
        return {"kind": kind, "rule": rule, "seq": seq, "d": d,
                "problems": _log(rng, 1, min(512, (262144 if d < 128 else 16384) // seq)),
                "store_s": d == 128 or rule == "delta" or rng.random() < 0.5}
    if kind == "swa":
        seq, heads = _log(rng, 48, 8192), rng.choice((4, 8, 16))
        return {"kind": kind, "batch": _log(rng, 1, max(1, min(16, 65536 // seq))), "heads": heads, "seq": seq,
                "hd": rng.choice((64, 64, 64, 64, 128)), "window": rng.choice((64, 128, 256, 512, 512))}
    if kind == "mlp":
        seq = _log(rng, 16, 384)
        d, hidden = rng.choice(((64, 256), (64, 256), (32, 128)))
        return {"kind": kind, "seq": seq, "problems": _log(rng, 2, min(148, 32768 // seq)), "d": d, "hidden": hidden,
                "activation": rng.choice((0, 0, 1, 2))}
    return {"kind": kind, "params": _log(rng, 20_000, 60_000_000), "tensors": rng.randint(4, 200)}


# ── inputs ─────────────────────────────────────────────────────────────────
class _Rand:
    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(self, *shape):
        return torch.randn(*shape, generator=self.g, device="cuda")

    def unit(self, *shape):
        return F.normalize(self.normal(*shape), dim=-1)

    def uniform(self, *shape):
        return torch.rand(*shape, generator=self.g, device="cuda")

    def zipf(self, vocab, *shape):
        """Zipf(1.1) token ids, the usual stand-in for text."""
        cdf = torch.cumsum(torch.arange(1, vocab + 1, device="cuda", dtype=torch.float64) ** -1.1, 0)
        return torch.searchsorted(cdf / cdf[-1], self.uniform(*shape).double()).clamp_(max=vocab - 1)


def _rule_inputs(c, seed):
    """Keys and queries L2-normalised; gates as the model's initial biases give them (retention
    gate sigmoid(3 + x), inner learning rate softplus(x - 4.6), momentum sigmoid(1.5 + x)); a carried
    memory and a momentum that starts from zero."""
    r = _Rand(seed)
    n, s, d = c["problems"], c["seq"], c["d"]
    st = dict(k=r.unit(n, s, d), v=r.normal(n, s, d) / math.sqrt(d), q=r.unit(n, s, d), dy=r.normal(n, s, d),
              alpha=torch.sigmoid(r.normal(n, s) + 3.0), theta=F.softplus(r.normal(n, s) - 4.6),
              eta=torch.sigmoid(r.normal(n, s) + 1.5), m0=0.1 * r.normal(n, d * d),
              s0=torch.zeros(n, d * d, device="cuda"))
    return st


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("exact", "chunkwise"):
        return dict(case=case, **_rule_inputs(case, seed))
    r = _Rand(seed)
    if kind == "model":
        cfg = StackedMAGConfig(d_model=case["d_model"], num_heads=case["heads"], n_blocks=case["blocks"],
                               seq_len=case["seq"])
        model = StackedMAG(cfg, case["batch"], device="cuda", seed=seed % (1 << 30) + 1)
        ids = r.zipf(cfg.vocab, case["batch"], case["seq"] + 1)
        st = dict(case=case, model=model, tokens=ids[:, :-1].contiguous(), targets=ids[:, 1:].contiguous())
        model.step_graphed(st["tokens"], st["targets"])      # a training program captures its step once
        return st
    if kind == "single":
        d, vocab = case["d_model"], case["vocab"]
        xav = lambda *sh: (2.0 * r.uniform(*sh) - 1.0) * math.sqrt(6.0 / sum(sh))
        p = {n: xav(d, d) for n in ("w_q", "w_k", "w_v", "w_o", "w_k_mem", "w_v_mem", "w_q_mem")}
        p.update(w_embed=r.normal(vocab, d), w_unembed=xav(d, vocab))
        for gate, bias in (("alpha", 3.0), ("theta", -4.6), ("eta", 1.5)):
            if gate != "eta" or case["rule"] == "titans":
                p["w_" + gate] = r.normal(2 * d) / math.sqrt(2 * d)
                p["b_" + gate] = torch.full((1,), bias, device="cuda")
        ids = (r.uniform(case["batch"], case["seq"] + 1) * vocab).long().clamp_(max=vocab - 1)
        return dict(case=case, model=MAGSingle(p, case["heads"], case["window"], case["rule"]),
                    ids=ids[:, :-1].contiguous(), targets=ids[:, 1:].contiguous())
    if kind == "swa":
        sh = (case["batch"], case["seq"], case["heads"] * case["hd"])
        mk = lambda: r.normal(*sh).bfloat16()
        return dict(case=case, q=mk(), k=mk(), v=mk(), do=r.normal(*sh))
    if kind == "mlp":
        n, s, d, dh = case["problems"], case["seq"], case["d"], case["hidden"]
        ss = D.mlp_state_size(d, dh)
        return dict(case=case, k=r.unit(n, s, d), v=0.5 * r.normal(n, s, d), q=r.unit(n, s, d), dy=r.normal(n, s, d),
                    alpha=torch.sigmoid(r.normal(n, s) - 3.0), theta=F.softplus(r.normal(n, s) - 4.6),
                    eta=torch.sigmoid(r.normal(n, s) + 1.5), m0=0.1 * r.normal(n, ss),
                    s0=torch.zeros(n, ss, device="cuda"))
    # adamw: a few large matrices and many small tensors, as the parameters of a model are
    nt = case["tensors"]
    share = [1.0 / (1 + i) for i in range(nt)]
    sizes = [max(1, int(case["params"] * x / sum(share))) for x in share]
    opt = FlatAdamW(sizes, device="cuda")
    opt.w.copy_(0.02 * r.normal(opt.arena_len))
    opt.g.copy_(0.01 * r.normal(opt.arena_len))
    return dict(case=case, opt=opt, step=0)


# ── one pass ───────────────────────────────────────────────────────────────
def run(st):
    c = st["case"]
    kind = c["kind"]
    if kind == "model":
        m = st["model"]
        loss = m.step_graphed(st["tokens"], st["targets"])
        return dict(loss=loss, w=m.opt.w, m=m.opt.m, v=m.opt.v, context=m.context)
    if kind == "single":
        loss, grads = st["model"].loss_and_grads(st["ids"], st["targets"])
        return dict(loss=loss, **grads)
    if kind == "swa":
        out, lse = D.swa_forward_lse(st["q"], st["k"], st["v"], c["heads"], c["hd"], c["window"])
        dq, dk, dv = D.swa_backward_lse(st["q"], st["k"], st["v"], out, lse, st["do"], c["heads"], c["hd"], c["window"])
        return dict(out=out, lse=lse, dq=dq, dk=dk, dv=dv)
    if kind == "adamw":
        opt = st["opt"]
        st["step"] += 1
        norm = opt.step(3e-4, [st["step"]] * len(opt.sizes), max_grad_norm=1.0)
        return dict(w=opt.w, m=opt.m, v=opt.v, norm=norm)
    k, v, q, al, th, et, m0, s0, dy = (st[n] for n in ("k", "v", "q", "alpha", "theta", "eta", "m0", "s0", "dy"))
    if kind == "mlp":
        ms, ss, y = D.titans_mlp_forward_dd(k, v, q, al, th, et, m0, s0, c["hidden"], c["activation"])
        g = D.titans_mlp_backward_dd(k, v, q, al, th, et, ms, ss, dy, c["hidden"], c["activation"])
        return dict(ms=ms, ss=ss, y=y, **g)
    if kind == "exact":
        if c["rule"] == "titans":
            ms, ss, y = D.titans_forward_dd(k, v, q, al, th, et, m0, s0, store_s=c["store_s"])
            return dict(ms=ms, ss=ss, y=y, **D.titans_backward_dd(k, v, q, al, th, et, ms, ss, dy))
        ms, y = D.delta_forward_dd(k, v, q, al, th, m0)
        return dict(ms=ms, y=y, **D.delta_backward_dd(k, v, q, al, th, ms, dy))
    if c["rule"] == "titans":
        mc, sc, y = D.titans_chunkwise_forward_dd(k, v, q, al, th, et, m0, s0, c["chunk"])
        return dict(mc=mc, sc=sc, y=y, **D.titans_chunkwise_backward_dd(k, v, q, al, th, et, mc, sc, dy, c["chunk"]))
    mc, y = D.delta_chunkwise_forward_dd(k, v, q, al, th, m0, c["chunk"])
    return dict(mc=mc, y=y, **D.delta_chunkwise_backward_dd(k, v, q, al, th, mc, dy, c["chunk"]))


# ── what a pass cannot do without ──────────────────────────────────────────
def work(case):
    kind = case["kind"]
    if kind in ("exact", "chunkwise"):
        n, s, d = case["problems"], case["seq"], case["d"]
        titans = case["rule"] == "titans"
        states = s + 1 if kind == "exact" else -(-s // case["chunk"]) + 1
        mats = 2 if titans and case.get("store_s", True) else 1
        io = n * s * (4 * d + 4 * d + 2 * (3 if titans else 2)) * 4      # k,v,q,dy in; y,dk,dv,dq out; gates both ways
        carry = (2 if titans else 1) * n * d * d * 4
        # forward: M k, state update, M q; backward: the two products again and their adjoints
        flops = n * s * d * d * ((8 + 22) if titans else (7 + 18))
        return {"bytes": io + carry + mats * n * states * d * d * 4, "flops": flops}
    if kind == "model":
        b, s, d, vocab, blocks, h = case["batch"], case["seq"], case["d_model"], 8192, case["blocks"], case["heads"]
        tok, hd = b * s, case["d_model"] // case["heads"]
        levels = sum(1.0 / min(c, s) for c in (1, 8, 64, 512))
        gemm = blocks * (4 * d * d + levels * 3 * d * d) + vocab * d
        window = min(512, s)
        pairs = b * h * (s * window - window * (window - 1) // 2)
        rule = blocks * levels * tok * h * hd * hd * 30
        params = 2 * vocab * d + blocks * (4 * d * d + 4 * (3 * d * d + 6 * d + 3) + 4 * d + 4) + 2 * d
        return {"bytes": 24 * params + 16 * tok + 2 * 4 * blocks * 4 * b * h * hd * hd,
                "flops": 6 * gemm * tok + 14 * hd * pairs * blocks + rule}
    if kind == "single":
        b, s, d, vocab = case["batch"], case["seq"], case["d_model"], case["vocab"]
        w = min(case["window"], s)
        pairs = b * (s * w - w * (w - 1) // 2)
        params = 7 * d * d + 2 * vocab * d
        return {"bytes": 8 * params + 16 * b * s,
                "flops": 6 * b * s * (7 * d * d + vocab * d) + 14 * d * pairs + 30 * b * s * d * d}
    if kind == "swa":
        b, h, s, hd, w = (case[n] for n in ("batch", "heads", "seq", "hd", "window"))
        w = min(w, s)
        e = b * s * h * hd
        return {"bytes": e * (4 * 2 + 4 + 3 * 4) + 4 * b * h * s,
                "flops": 14 * hd * b * h * (s * w - w * (w - 1) // 2)}
    if kind == "mlp":
        n, s, d, dh = case["problems"], case["seq"], case["d"], case["hidden"]
        ss = D.mlp_state_size(d, dh)
        return {"bytes": n * s * (8 * d + 6) * 4 + 2 * n * ss * 4 + 2 * n * (s + 1) * ss * 4,
                "flops": n * s * ss * 40}
    return {"bytes": case["params"] * 28, "flops": case["params"] * 16}


def tolerance(case):
    kind = case["kind"]
    if kind == "model":
        # bf16 activations and weights; v holds squares of gradients
        return {"rel": 1e-2, "max": 0.5}
    if kind == "swa":
        return {"rel": 1e-2}                        # bf16 operands
    if kind == "adamw":
        return {"rel": 1e-5}
    # fp32 recurrences over hundreds to thousands of chained tokens; the momentum gate's gradient is
    # a difference of states divided by the gate where only one trajectory is stored
    return {"rel": 1e-4 if kind == "mlp" else 3e-5, "max": 2e-3}
