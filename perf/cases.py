"""Workloads of the attention op that stand for its real use, for timing and for comparing results.

Every case is one call of a public function of `flash_msa_b200` on tensors that are already on the GPU: a training pass
(forward, then backward into all five inputs) or a forward pass alone (evaluation).  Sizes are those of the benchmark
configurations, of the reference project's own test and sweep defaults, and of the tests in this repository.
"""
import math

import numpy as np
import torch

import flash_msa_b200 as fm

BLOCK = 128
D = 128
SCALE = D ** -0.5

_DEFAULTS = dict(path="sparse", train=True, kl=True, dtype="bf16", layout="bhsd", docs=0, sinks=False, skew=False)


def _case(**kw):
    return dict(_DEFAULTS, **kw)


def listed():
    return [
        # The smallest call: evaluation of a toy model.  Latency of the host path and of the launches.
        _case(name="forward_s512", b=1, s=512, hq=4, hkv=1, hp=2, hpkv=1, kb=2, train=False),
        # Configuration 1: one short sequence, the size at which a user first tries the op.
        _case(name="train_s1024_top4", b=1, s=1024, hq=8, hkv=2, hp=2, hpkv=2, kb=4),
        # The defaults of the reference project's own tests, with activations as its model passes them: views of (B,S,H,D).
        _case(name="train_s2048_top4", b=1, s=2048, hq=16, hkv=2, hp=4, hpkv=1, kb=4, layout="bshd"),
        # Odd sizes: 13 blocks, five main heads per proxy head, three sequences; fp16, softmax sinks, a frozen selector (no
        # gradient reaches the KL loss).
        _case(name="train_s1664_fp16_sinks", b=3, s=1664, hq=20, hkv=2, hp=4, hpkv=2, kb=5, dtype="fp16", sinks=True, kl=False),
        # The largest shape of the reference project's training sweep.
        _case(name="train_s4096_top16", b=4, s=4096, hq=16, hkv=2, hp=4, hpkv=1, kb=16, layout="bshd"),
        # Configuration 2, the headline: 8K training, and the same shape in evaluation (prefill).
        _case(name="train_s8192_top16", b=2, s=8192, hq=32, hkv=8, hp=8, hpkv=8, kb=16),
        _case(name="forward_s8192_top16", b=2, s=8192, hq=32, hkv=8, hp=8, hpkv=8, kb=16, train=False),
        # 8K training on packed documents whose boundaries fall inside blocks.
        _case(name="train_s8192_packed", b=1, s=8192, hq=32, hkv=8, hp=8, hpkv=8, kb=16, docs=5),
        # Configuration 3: the warmup stage, dense attention and the KL loss over the full sequence.
        _case(name="warmup_s4096", path="warmup", b=4, s=4096, hq=32, hkv=8, hp=8, hpkv=8, kb=16),
        # More than 64 selected blocks per row and twelve main heads per proxy head.
        _case(name="train_s16384_top96", b=1, s=16384, hq=24, hkv=2, hp=2, hpkv=1, kb=96),
        # Configuration 5 as one of eight GPUs sees it: one KV group of a 64K sequence.
        _case(name="train_s65536_top32", b=1, s=65536, hq=8, hkv=1, hp=2, hpkv=1, kb=32),
        # Configuration 4, one sequence: 64 blocks per row, block-mean keys, sharp block scores, sink blocks.
        _case(name="train_s32768_skewed", b=1, s=32768, hq=48, hkv=4, hp=8, hpkv=4, kb=64, skew=True),
    ]


def _tile_rows(c):
    """(query row, head, key block) triples the path visits: the measure of a case's size."""
    nb = c["s"] // BLOCK
    per_row = (nb + 1) / 2 if c["path"] == "warmup" else c["kb"]
    return c["b"] * c["hq"] * c["s"] * per_row


def draw(rng):
    """A case of the ranges above: lengths from 256 to 64K in steps of a block, one to eight KV heads, one to twelve main
    heads per proxy head, up to 96 selected blocks, every option."""
    while True:
        path = "warmup" if rng.random() < 0.2 else "sparse"
        longest = 8192 if path == "warmup" else 65536
        s = BLOCK * int(round(math.exp(rng.uniform(math.log(2), math.log(longest // BLOCK)))))
        nb = s // BLOCK
        hkv = rng.choice([1, 2, 3, 4, 8])
        hp = hkv * rng.choice([1, 1, 2])
        hpkv = rng.choice([1, hkv, hp])
        c = _case(path=path, b=rng.choice([1, 1, 2, 3, 4]), s=s, hq=hp * rng.choice([1, 2, 3, 4, 4, 5, 6, 8, 12]), hkv=hkv, hp=hp,
                  hpkv=hpkv, kb=min(nb, int(round(math.exp(rng.uniform(math.log(1.5), math.log(96)))))))
        c["train"] = rng.random() < 0.75
        c["kl"] = rng.random() < 0.75
        c["dtype"] = "fp16" if rng.random() < 0.25 else "bf16"
        c["layout"] = rng.choice(["bhsd", "bshd"])
        c["docs"] = rng.randint(2, min(12, nb)) if rng.random() < 0.25 else 0
        c["sinks"] = rng.random() < 0.15
        c["skew"] = rng.random() < 0.25
        if _tile_rows(c) <= 6e7 and c["b"] * c["hq"] * c["s"] <= 2.5e6:
            return c


def _documents(case):
    """Boundaries of the packed documents: lengths of some spread, not multiples of a block."""
    if not case["docs"]:
        return None
    w = np.random.RandomState(case["s"] + case["docs"]).uniform(0.5, 1.5, case["docs"])
    cuts = np.unique(np.round(np.cumsum(w)[:-1] / w.sum() * case["s"]).astype(int))
    return [0] + [int(x) for x in cuts if 0 < x < case["s"]] + [case["s"]]


def prepare(case, seed):
    dev = torch.device("cuda")
    dtype = torch.float16 if case["dtype"] == "fp16" else torch.bfloat16
    gen = torch.Generator(device=dev).manual_seed(seed)
    b, s, hq, hkv, hp, hpkv = (case[n] for n in ("b", "s", "hq", "hkv", "hp", "hpkv"))
    nb = s // BLOCK

    def normal(*shape):
        return torch.randn(*shape, generator=gen, device=dev)

    qp, kp, q, k, v = (normal(b, h, s, D) for h in (hp, hpkv, hq, hkv, hkv))
    if case["skew"]:
        sink_rng = np.random.RandomState(seed % (1 << 31))
        sink_blocks = [sink_rng.choice(nb, min(4, nb), replace=False) for _ in range(b)]
        for t, h in ((k, hkv), (kp, hpkv)):
            t4 = t.view(b, h, nb, BLOCK, D)
            t4.mul_(0.5).add_(normal(b, h, nb, 1, D))
            for i in range(b):
                t4[i, :, torch.as_tensor(sink_blocks[i], device=dev)] *= 3.0
        qp *= 4.0

    def finish(t):   # (B,H,S,D) in the case's type and layout
        t = t.to(dtype)
        return t.transpose(1, 2).contiguous().transpose(1, 2) if case["layout"] == "bshd" else t

    state = {"inputs": [finish(t) for t in (qp, kp, q, k, v)], "top_k": case["kb"] * BLOCK, "train": case["train"],
             "warmup": case["path"] == "warmup", "cu_seqlens": _documents(case), "sinks": None, "kl": case["kl"]}
    if case["sinks"]:
        state["sinks"] = normal(hq) * 0.7 + 0.5
    if case["train"]:
        state["d_out"] = normal(b, s, hq * D).to(dtype)
        state["d_kl"] = torch.ones((), device=dev)
    return state


def _attend(state, tensors, sinks):
    if state["cu_seqlens"] is not None:
        fn = fm.flash_msa_warmup_varlen_func if state["warmup"] else fm.flash_msa_varlen_func
        return fn(*tensors, state["cu_seqlens"], state["top_k"], SCALE, sinks=sinks)
    fn = fm.flash_msa_warmup_func if state["warmup"] else fm.flash_msa_func
    return fn(*tensors, state["top_k"], SCALE, sinks=sinks)


def run(state):
    if not state["train"]:
        with torch.no_grad():
            out, _ = _attend(state, state["inputs"], state["sinks"])
        return {"out": out}
    leaves = [t.detach().requires_grad_(True) for t in state["inputs"]]
    sinks = None if state["sinks"] is None else state["sinks"].detach().requires_grad_(True)
    out, kl = _attend(state, leaves, sinks)
    if state["kl"]:
        torch.autograd.backward([out, kl], [state["d_out"], state["d_kl"]])
    else:
        torch.autograd.backward([out], [state["d_out"]])
    grads = dict(zip(("dq_proxy", "dk_proxy", "dq", "dk", "dv"), (t.grad for t in leaves)))
    if sinks is not None:
        grads["dsinks"] = sinks.grad
    return {"out": out.detach(), **grads}


def _pairs(case):
    """((query, key) pairs per head that the main attention needs, pairs whose block scores the selection needs), per batch
    element."""
    s = case["s"]
    q = np.arange(s, dtype=np.int64)
    cu = np.asarray(_documents(case) or [0, s])
    lo = cu[np.searchsorted(cu, q, side="right") - 1]          # first token of the row's document
    visible = q - lo + 1
    if case["path"] == "warmup":
        return int(visible.sum()), 0
    own = q - np.maximum(lo, q // BLOCK * BLOCK) + 1
    picked = np.minimum(visible, own + (case["kb"] - 1) * BLOCK)
    return int(picked.sum()), int((visible - own).sum())


def work(case):
    b, s, hq, hkv, hp, hpkv = (case[n] for n in ("b", "s", "hq", "hkv", "hp", "hpkv"))
    hp_eff = max(hp, hkv)
    main, scored = _pairs(case)
    product = 2 * D
    proxy = case["train"] and case["kl"]
    flops = product * b * (scored * hp + main * hq * (7 if case["train"] else 2))
    if proxy:   # the proxy's log-sum-exp and its three gradient products
        flops += product * b * main * hp_eff * 4
    row = b * s * D * 2
    inputs = row * (hq + 2 * hkv)
    if case["path"] != "warmup" or proxy:
        inputs += row * (hp + hpkv)
    if case["train"]:   # d_out comes in; out and five gradients leave
        nbytes = inputs + row * hq + row * (2 * hq + 2 * hkv + hp + hpkv)
    else:
        nbytes = inputs + row * hq
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Products of 16-bit operands, 16-bit probabilities and score gradients between the products, 16-bit results."""
    return {"rel": 4e-3 if case["dtype"] == "fp16" else 1e-2}
