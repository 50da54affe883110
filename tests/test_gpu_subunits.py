"""How a launch is cut into sub-units must not show in its results: one pass over all (batch, KV head) groups against one pass per
group, whose launches take other sub-unit lengths and finer last groups."""
import pytest
import torch

from tests.gpu_util import SCALE, bf16_inputs, forward_tiles, max_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,s,kb,docs,form", [
    (1, 4096, 16, False, None), (2, 4096, 16, False, None), (4, 4096, 16, True, None), (5, 4096, 16, False, None), (3, 1664, 5, True, None),
    (2, 8192, 2, False, "four"), (2, 8192, 3, False, "shared"), (2, 8192, 3, True, "four"), (1, 12544, 4, True, "shared fp16")])
def test_one_pass_against_a_pass_per_group(monkeypatch, b, s, kb, docs, form):
    """The backward with sub-units of 2, 4, 8 and 16 chunks at most in the one pass (and 1, rows that end inside a chunk, in the case of
    1664); in the cases with a `form` (four KV heads, or three with two proxy heads each) also the forward, whose key-block stationary
    kernels then work on the tiles that the other one leaves."""
    import flash_msa_b200 as fm
    from flash_msa_b200 import ops
    heads = dict(hq=12, hkv=3, hp=6, hpkv=3) if form and form.startswith("shared") else dict(hq=4, hkv=4, hp=4, hpkv=4)
    dt = torch.float16 if form == "shared fp16" else torch.bfloat16
    *inputs, do = bf16_inputs(dict(b=b, s=s, seed=b + s, **heads), dtype=dt)
    tiles = forward_tiles(inputs, kb, [0, s // 3, s // 2 + 5, s] if docs else None)
    assert 1 <= tiles < s // 128 if form else tiles == s // 128
    kl_weight = torch.tensor(float(s if dt == torch.float16 else 1), device="cuda")   # (proxy gradients above fp16's subnormals)
    res = []
    for cap in (None, 1):
        if cap:
            monkeypatch.setattr(ops, "MAX_PARTIAL_BYTES", cap)
        leaves = [t.detach().requires_grad_(True) for t in inputs]
        if docs:
            out, kl = fm.flash_msa_varlen_func(*leaves, [0, s // 3, s // 2 + 5, s], kb * 128, SCALE)
        else:
            out, kl = fm.flash_msa_func(*leaves, kb * 128, SCALE)
        torch.autograd.backward([out, kl], [do, kl_weight])
        res.append([out] + [t.grad for t in leaves])
    for n, a, c in zip(["out", "dq_proxy", "dk_proxy", "dq", "dk", "dv"], *res):
        # (the order in which sub-units add to dK, dV and dKp is free: the last bit of the 16-bit result)
        assert max_err(a, c) <= (0.0 if n in ("out", "dq", "dq_proxy") else 2 ** -7 * c.float().abs().max().item()), n


@pytest.mark.parametrize("b,s,hkv,kb,docs", [(1, 12544, 2, 2, True), (2, 12544, 1, 3, False), (1, 33024, 1, 1, False)])
def test_few_blocks_of_a_long_sequence(b, s, hkv, kb, docs):
    """Most sub-units lie beyond the end of their rows, more than the 32 that a draw looks at.  With values and dO of one every output is
    one, and a (batch, KV head)'s dV sums to its number of query rows; a chunk left out or taken twice would move that by more than
    64 / s >= 2^-9 of it.  Rounded weights and results, each off by 2^-9 at most and in no direction, move the sum of 128 kb terms per row
    and s rows by 2^-9 / sqrt(s) of it."""
    import flash_msa_b200 as fm
    (qp, kp, q, k, v), do = (lambda x: (x[:-1], x[-1]))(bf16_inputs(dict(b=b, s=s, hq=2 * hkv, hkv=hkv, hp=hkv, hpkv=hkv, seed=s + kb)))
    leaves = [t.detach().requires_grad_(True) for t in (qp, kp, q, k, torch.ones_like(v))]
    if docs:
        out, kl = fm.flash_msa_varlen_func(*leaves, [0, s // 3, s // 2 + 5, s], kb * 128, SCALE)
    else:
        out, kl = fm.flash_msa_func(*leaves, kb * 128, SCALE)
    out.backward(torch.ones_like(do))
    # weights and partial outputs rounded to 16 bits, 2^-9 each, then the result, half of bf16's step of 2^-7 above one: 2^-7
    assert (out.float() - 1).abs().max().item() <= 2 ** -7
    total = leaves[4].grad.double().sum(-2 if leaves[4].shape[2] == s else 1)
    assert (total / (2 * s) - 1).abs().max().item() <= 2 ** -11
