"""The query-tile stationary forward against the key-block stationary one (a reverse index without its selection sends every
tile the general way): sizes at which tiles, words of the visit lists and the ring of items end, every layout, type and mask."""
import dataclasses

import pytest
import torch

from oracle import msa_oracle as O
from tests.gpu_util import SCALE, bf16_inputs, kernel_selection, max_err, yardstick_check

pytestmark = pytest.mark.gpu


def _selection(cfg, kind):
    """int32 [B,Hp,S,Kb]: own block, then `kind` of the others, the sentinel NB where there are no more."""
    b, hp, s, kb = cfg["b"], cfg["hp"], cfg["s"], cfg["kb"]
    nb = s // 128
    own = (torch.arange(s) // 128).view(1, 1, s, 1)
    g = torch.Generator().manual_seed(s + kb)
    key = torch.rand(b, hp, s, nb, generator=g)
    if kind == "alike":    # the rows of a tile agree but for a few, so that most blocks are visited by no row or by all of them
        key = torch.where(torch.rand(b, hp, s, 1, generator=g) < 0.02, key, key[:, :, ::128].repeat_interleave(128, 2))
    key = key.masked_fill(torch.arange(nb).view(1, 1, 1, nb) > own, -1.0).scatter(3, own.expand(b, hp, s, 1), 2.0)
    val, idx = key.sort(dim=-1, descending=True)
    return torch.where(val >= 0, idx, nb)[..., :kb].to(torch.int32).contiguous().cuda()


CFGS = [
    dict(b=1, s=128, hq=1, hkv=1, hp=1, hpkv=1, kb=1),
    dict(b=3, s=256, hq=6, hkv=1, hp=2, hpkv=1, kb=1),
    dict(b=2, s=640, hq=12, hkv=2, hp=4, hpkv=2, kb=3),
    dict(b=1, s=4224, hq=5, hkv=1, hp=1, hpkv=1, kb=20),     # 33 blocks: a second round of 32 in the list of visited blocks
    dict(b=1, s=8448, hq=4, hkv=2, hp=2, hpkv=2, kb=40),     # 66 blocks, all tiles
    dict(b=1, s=8448, hq=4, hkv=1, hp=2, hpkv=1, kb=3),      # the first six tiles, the others the general way
    dict(b=2, s=4096, hq=24, hkv=2, hp=2, hpkv=1, kb=2),     # ... with twelve heads per proxy head
]


@pytest.mark.parametrize("kind", ["random", "alike"])
@pytest.mark.parametrize("cfg", CFGS, ids=lambda c: f"s{c['s']}_kb{c['kb']}_mpp{c['hq'] // c['hp']}")
@pytest.mark.parametrize("form", ["plain", "fp16", "bshd", "docs"])
def test_agrees_with_the_key_block_stationary_forward(cfg, kind, form):
    from flash_msa_b200 import _lib, ops
    dt = torch.float16 if form == "fp16" else torch.bfloat16
    qp, kp, q, k, v, _ = bf16_inputs(dict(cfg, seed=cfg["s"]), layout="bshd" if form == "bshd" else "bhsd", dtype=dt)
    qp = qp * 3   # sharper proxy rows: their maxima rise by more than the lazy rescale lets pass
    if form != "bshd":
        q = q * 4
    cu = [0, cfg["s"] // 3, cfg["s"] // 3 + 1, cfg["s"]] if form == "docs" else None
    ds = None if cu is None else ops.doc_start_from_cu_seqlens(cu, cfg["b"], cfg["s"], q.device)
    idx = _selection(cfg, kind)
    if ds is not None:   # a selection never holds blocks that end before the row's document
        idx = torch.where(idx < (ds // 128).view(cfg["b"], 1, -1, 1), cfg["s"] // 128, idx)
    rix = ops.build_reverse_index(idx)
    pb = ops._problem(q, k, qp, kp, cfg["kb"], SCALE)
    assert 1 <= _lib.load().fmsa_forward_tiles(pb, 0, 0) <= cfg["s"] // 128
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    got = ops.attention_forward(q, k, v, qp, kp, SCALE, rix, doc_start=ds, status=status)
    want = ops.attention_forward(q, k, v, qp, kp, SCALE, dataclasses.replace(rix, block_indices=None), doc_start=ds, status=status)
    ops.check_status(status, "forward")
    # Both round P and the result to 16 bits (u = 2^-9 or 2^-12 of an element, P weighted with |v|), one of them the partial rows as
    # well: five such errors of at most u max|v|.  The logarithms are those of fp32 sums of the same exponentials (2^-22 each).
    u = 2.0 ** (-12 if dt == torch.float16 else -9)
    assert max_err(got[0], want[0]) <= 5 * u * v.float().abs().max().item()
    assert max_err(got[1], want[1]) <= 1e-4 and max_err(got[2], want[2]) <= 1e-4
    alone = ops.attention_forward(q, k, v, qp, kp, SCALE, rix, doc_start=ds, with_proxy=False)
    assert torch.equal(alone[0], got[0]) and torch.equal(alone[1], got[1])


@pytest.mark.parametrize("s,kb", [(384, 2), (8192, 1)])
def test_sinks_in_both_forwards(s, kb):
    """All tiles, and the first two of 64, whose log-sum-exps take the sinks in different kernels."""
    import flash_msa_b200 as fm
    cfg = dict(b=1, s=s, hq=4, hkv=1, hp=1, hpkv=1, kb=kb, seed=5)
    qp, kp, q, k, v, do = bf16_inputs(cfg)
    sinks = torch.tensor([-3.0, 0.0, 2.0, 6.0], device="cuda", requires_grad=True)
    leaves = [t.detach().requires_grad_(True) for t in (qp, kp, q, k, v)]
    out, kl = fm.flash_msa_func(*leaves, kb * 128, SCALE, sinks=sinks)
    torch.autograd.backward([out, kl], [do, torch.ones((), device="cuda")])
    with torch.no_grad():
        alone, _ = fm.flash_msa_func(qp, kp, q, k, v, kb * 128, SCALE, sinks=sinks)
    assert torch.equal(alone, out)
    idx = kernel_selection(qp, kp, kb)
    args = (qp, kp, q, k, v, kb * 128, SCALE, do, 1.0)
    r32 = O.sparse_forward_backward(*args, block_indices=idx, sinks=sinks.detach())
    r16 = O.sparse_forward_backward(*args, block_indices=idx, sinks=sinks.detach(), dtype=torch.bfloat16)
    yardstick_check("out", out, r32["out"], r16["out"], 2e-3)
    for n, leaf in zip(["dq_proxy", "dk_proxy", "dq", "dk", "dv"], leaves):
        yardstick_check(n, leaf.grad, r32[n], r16[n], 2e-3 * r32[n].abs().max().item())


@pytest.mark.parametrize("s,kb,cu", [(8192, 2, list(range(0, 8192, 500)) + [8192]), (8448, 4, [0, 0, 1200, 2400, 3700, 3701, 5000, 6200, 7400, 8448])])
def test_short_documents(s, kb, cu):
    """Boundaries that the host knows to be close send all tiles the query-tile stationary way, the same ones in device memory only
    the first; errors as above."""
    import flash_msa_b200 as fm
    cfg = dict(b=2, s=s, hq=8, hkv=2, hp=2, hpkv=1, seed=s)
    qp, kp, q, k, v, do = bf16_inputs(cfg)
    res = []
    for bounds in (cu, torch.tensor(cu, device="cuda")):
        leaves = [t.detach().requires_grad_(True) for t in (qp, kp, q, k, v)]
        out, kl = fm.flash_msa_varlen_func(*leaves, bounds, kb * 128, SCALE)
        torch.autograd.backward([out, kl], [do, torch.ones((), device="cuda")])
        with torch.no_grad():
            alone, _ = fm.flash_msa_varlen_func(qp, kp, q, k, v, bounds, kb * 128, SCALE)
        assert torch.equal(alone, out)
        res.append([out] + [t.grad for t in leaves])
    assert max_err(res[0][0], res[1][0]) <= 5 * 2.0 ** -9 * v.float().abs().max().item()
    for n, a, b in zip(["dq_proxy", "dk_proxy", "dq", "dk", "dv"], res[0][1:], res[1][1:]):
        assert max_err(a, b) <= 2e-2 * b.float().abs().max().item(), n   # (delta is formed from the 16-bit output)


def test_rows_that_select_nothing():
    """Not what a selection gives, but what the index accepts: no edge for some rows, for a whole tile of them, or for all."""
    from flash_msa_b200 import ops
    cfg = dict(b=1, s=512, hq=4, hkv=2, hp=2, hpkv=1, kb=2, seed=3)
    qp, kp, q, k, v, _ = bf16_inputs(cfg)
    idx = _selection(cfg, "random")
    idx[:, 0, 100:300] = 4
    idx[:, 1, 384:] = 4
    out, lse, lse_p = ops.attention_forward(q, k, v, qp, kp, SCALE, ops.build_reverse_index(idx))
    none = (idx == 4).all(-1)                                    # [B,Hp,S]
    rows = none.repeat_interleave(2, 1)                          # of the main heads
    heads = out.view(1, 512, 4, 128).transpose(1, 2)
    assert (heads[rows] == 0).all() and torch.isneginf(lse[rows]).all() and torch.isneginf(lse_p[none]).all()
    assert torch.isfinite(lse[~rows]).all() and torch.isfinite(out).all()


@pytest.mark.parametrize("sinks", [False, True])
@pytest.mark.parametrize("gap", [-5.7, -5.4, 12.0, 14.0, 16.0])
def test_fp16_probabilities_far_below_the_maximum(gap, sinks):
    """One key of the block visited first lies `gap` above the N(0,1) logits of the others and has a value of zero, so that the rows of
    that tile are sums of small probabilities; the other way round (-5.4, 7.8 in the log2 domain, and -5.7), all of the second block
    just below and above the line at which O is rescaled.  Independent roundings of P, normal (2^-11) or of the subnormals below 2^-21 of the
    maximum (2^-25 at most, against a root mean square of e 2^-16 at a gap of 16: 4e-4), and of the result (2^-11) add up to less than
    1e-3 in the 2-norm."""
    import flash_msa_b200 as fm
    s, h = 4096, 2
    g = torch.Generator().manual_seed(21)
    qp, kp = (torch.randn(1, 1, s, 128, generator=g).half().cuda() for _ in range(2))
    q, k, v = (torch.randn(1, h, s, 128, generator=g) for _ in range(3))
    v *= 256   # (no subnormal results)
    q[..., 0], k[..., 0] = 4.0, 0.0
    if gap > 0:
        k[:, :, s - 128] = 0
        k[:, :, s - 128, 0] = gap / (4.0 * SCALE)
        v[:, :, s - 128] = 0
    else:
        k.zero_()
        k[:, :, s - 256:s - 128, 0] = -gap / (4.0 * SCALE)
    q, k, v = (t.half().cuda() for t in (q, k, v))
    bias = torch.tensor([2.0, gap + 1.0], device="cuda") if sinks else None
    with torch.no_grad():
        out, _ = fm.flash_msa_warmup_func(qp, kp, q, k, v, s, SCALE, sinks=bias)
    rows = slice(s - 128, s)
    logits = q[:, :, rows].double() @ k.double().transpose(2, 3) * SCALE
    hidden = torch.arange(s, device="cuda") > torch.arange(s - 128, s, device="cuda").view(-1, 1)
    logits = logits.masked_fill(hidden, -torch.inf)
    norm = logits.logsumexp(-1, keepdim=True)
    if sinks:
        norm = torch.logaddexp(norm, bias.double().view(1, h, 1, 1))
    want = (logits - norm).exp() @ v.double()
    got = out.view(1, s, h, 128).transpose(1, 2)[:, :, rows].double()
    assert ((got - want).norm(dim=(2, 3)) / want.norm(dim=(2, 3))).max() < 1e-3


@pytest.mark.parametrize("cap", [None, 1])
@pytest.mark.parametrize("cfg", [CFGS[0], *CFGS[-2:], dict(b=2, s=5120, hq=4, hkv=2, hp=4, hpkv=2, kb=1)], ids=lambda c: f"s{c['s']}_kb{c['kb']}")
def test_stages_of_the_tiles_behind(monkeypatch, cfg, cap):
    """The key-block stationary stages work on the query tiles behind the others' only, from the right place of every reverse-index
    row, and together they give the whole pass's output bit for bit, in one pass over the groups or several."""
    import flash_msa_b200 as fm
    from flash_msa_b200 import _lib, ops
    if cap:
        monkeypatch.setattr(ops, "MAX_PARTIAL_BYTES", cap)
    qp, kp, q, k, v, _ = bf16_inputs(dict(cfg, seed=7))
    b, hp, nb, s = cfg["b"], cfg["hp"], cfg["s"] // 128, cfg["s"]
    rix = ops.build_reverse_index(ops.select_blocks_fused(qp, kp, SCALE, cfg["kb"]))
    tiles = _lib.load().fmsa_forward_tiles(ops._problem(q, k, qp, kp, cfg["kb"], SCALE), 0, 0)
    lib, calls = _lib.load(), []

    class Recorder:
        def __getattr__(self, name):
            def call(*args):
                calls.append((name, args))
                return getattr(lib, name)(*args)
            return call
    monkeypatch.setattr(_lib, "load", Recorder)
    out, _, _ = ops.attention_forward(q, k, v, qp, kp, SCALE, rix)
    monkeypatch.undo()
    first = [a[8] for n, a in calls if n in ("fmsa_sparse_fwd_from", "fmsa_sparse_fwd_combine_from")]
    assert not any(n in ("fmsa_sparse_fwd", "fmsa_sparse_fwd_combine") for n, _ in calls)
    assert first == [] if tiles == nb else first and set(first) == {tiles}
    with torch.no_grad():
        want, _ = fm.flash_msa_func(qp, kp, q, k, v, cfg["kb"] * 128, SCALE)
    assert torch.equal(out, want)
    row_ptr, col_q = rix.row_ptr.cpu(), rix.col_q.cpu()
    for t in {0, 1, tiles, nb}:
        start = torch.empty(b * hp * nb, dtype=torch.int32, device="cuda")
        _lib.check(lib.fmsa_row_start(rix.row_ptr.data_ptr(), rix.col_q.data_ptr(), b * hp, s, t, start.data_ptr(),
                                      torch.cuda.current_stream().cuda_stream), "fmsa_row_start")
        ends = torch.tensor([int((col_q[row_ptr[r]:row_ptr[r + 1]] < 128 * t).sum()) for r in range(b * hp * nb)])
        assert torch.equal(start.cpu(), row_ptr[:-1] + ends)


@pytest.mark.parametrize("b,s,heads,form", [(2, 640, dict(hq=12, hkv=2, hp=4, hpkv=2), "docs"), (1, 1664, dict(hq=9, hkv=1, hp=1, hpkv=1), "plain"),
                                            (1, 2048, dict(hq=4, hkv=2, hp=2, hpkv=1), "fp16")])
def test_dense_schedule_of_the_key_block_stationary_stages(b, s, heads, form):
    """No call of the package takes a dense forward this way, but the two stages accept it: a pass over all groups and one per group against
    the query-tile stationary stage, with the errors of the first test above."""
    from flash_msa_b200 import _lib, ops
    dt = torch.float16 if form == "fp16" else torch.bfloat16
    qp, kp, q, k, v, _ = bf16_inputs(dict(b=b, s=s, seed=s, **heads), dtype=dt)
    ds = ops.doc_start_from_cu_seqlens([0, s // 3, s // 3 + 1, s], b, s, q.device) if form == "docs" else None
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    want = ops.attention_forward(q, k, v, qp, kp, SCALE, None, dense=True, doc_start=ds, status=status)
    lib, pb, st = _lib.load(), ops._problem(q, k, qp, kp, 1, SCALE, ds), torch.cuda.current_stream().cuda_stream
    args = [ops._tensor_arg(t) for t in (q, k, v, qp, kp)]
    mpp, groups = heads["hq"] // heads["hp"], b * heads["hkv"]
    u = 2.0 ** (-12 if dt == torch.float16 else -9)
    for step in (groups, 1):
        got = [torch.full_like(t, float("nan")) for t in want]
        slots = lib.fmsa_fwd_partial_slots(pb, step, 1)
        o_part = torch.empty(slots * mpp * 128, dtype=dt, device="cuda")
        stats = torch.empty(slots * (mpp + 1) * 2, dtype=torch.float32, device="cuda")
        counter = torch.empty(1, dtype=torch.int32, device="cuda")
        for g0 in range(0, groups, step):
            _lib.check(lib.fmsa_sparse_fwd(pb, *args, 0, 0, o_part.data_ptr(), stats.data_ptr(), slots, g0, step, 1, 1, counter.data_ptr(),
                                           status.data_ptr(), st), "fmsa_sparse_fwd")
            _lib.check(lib.fmsa_sparse_fwd_combine(pb, o_part.data_ptr(), stats.data_ptr(), 0, 0, *(t.data_ptr() for t in got), g0, step, 1, st),
                       "fmsa_sparse_fwd_combine")
        ops.check_status(status, "forward")
        assert max_err(got[0], want[0]) <= 5 * u * v.float().abs().max().item()
        assert max_err(got[1], want[1]) <= 1e-4 and max_err(got[2], want[2]) <= 1e-4
