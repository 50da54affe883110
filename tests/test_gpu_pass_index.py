"""The reverse index of a whole pass, whose counts come from the selection, against the one that counts the indices again, and what
the kernels behind a selection make of a tile that selects nothing (what a selection leaves that had to give a tile up)."""
import pytest
import torch

from oracle import msa_oracle as O
from tests.gpu_util import SCALE, bf16_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,hp,s,kb,docs", [
    (1, 1, 128, 1, False),
    (8, 8, 2048, 3, False),      # 1024 columns of 16, the most that one scan kernel takes
    (13, 5, 2048, 3, False),     # 1040 columns
    (16, 8, 1024, 8, True),      # 1024 columns of 8
    (43, 3, 1024, 2, False),     # 1032 columns of 8
    (1, 1, 16384, 5, False),     # one column of 128 per block: 16384 counts
    (1, 1, 16512, 5, True),      # 129 blocks, more counts than that
    (2, 3, 1664, 13, True),
])
def test_counts_of_the_selection(b, hp, s, kb, docs):
    from flash_msa_b200 import ops, passes
    cfg = dict(b=b, s=s, hq=hp, hkv=1, hp=hp, hpkv=1, seed=s + hp)
    inputs = bf16_inputs(cfg)[:5]
    qp, kp, q, _, _ = inputs
    ds = ops.doc_start_from_cu_seqlens([0, s // 3 + 5, s // 2, s], b, s, q.device) if docs else None
    plan = passes.plan(inputs, kb, SCALE, False)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    saved = passes.forward(plan, inputs, ds, None, status.data_ptr(), True)[2]
    ops.check_status(status, "forward")
    idx = ops.select_blocks_fused(qp, kp, SCALE, kb, doc_start=ds)
    rix = ops.build_reverse_index(idx)
    nb, at = s // 128, [a // 4 for a in plan.at]
    row_ptr = saved[at[0]:at[0] + b * hp * nb + 1]
    edges = int(row_ptr[-1])
    assert torch.equal(row_ptr, rix.row_ptr[:row_ptr.numel()])
    assert torch.equal(saved[at[1]:at[1] + edges], rix.col_q[:edges])
    assert torch.equal(saved[at[2]:at[2] + idx.numel()], rix.edge_pos.reshape(-1)[:idx.numel()])
    want = O.reverse_index(idx.cpu(), nb)
    for got, ref in zip((row_ptr, saved[at[1]:at[1] + edges], saved[at[2]:at[2] + idx.numel()]), want):
        assert torch.equal(got.cpu().to(ref.dtype), ref.reshape(-1)[:got.numel()])


@pytest.mark.parametrize("s,kb,tile", [(512, 2, 3), (512, 2, 0), (8192, 1, 1), (8192, 1, 40)])
def test_tiles_that_select_nothing(s, kb, tile):
    """Such a tile's rows have no sum to take a logarithm of and gradients of zero, and the others are as without it."""
    from flash_msa_b200 import ops
    cfg = dict(b=1, s=s, hq=4, hkv=2, hp=2, hpkv=1, seed=s + tile)
    qp, kp, q, k, v, do = bf16_inputs(cfg)
    whole = ops.select_blocks_fused(qp, kp, SCALE, kb)
    idx = whole.clone()
    rows = slice(128 * tile, 128 * tile + 128)
    idx[:, :, rows] = s // 128
    one = torch.ones((), device="cuda")
    res = []
    for sel in (whole, idx):
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        rix = ops.build_reverse_index(sel)
        out, lse, lse_p = ops.attention_forward(q, k, v, qp, kp, SCALE, rix, status=status)
        grads = ops.attention_backward(q, k, v, qp, kp, out, do, lse, lse_p, SCALE, rix, one, status=status)
        ops.check_status(status, "pass")
        res.append((out, lse, lse_p, grads))
    (out0, lse0, _, grads0), (out, lse, lse_p, grads) = res
    assert torch.isneginf(lse[:, :, rows]).all() and torch.isneginf(lse_p[:, :, rows]).all()
    keep = torch.ones(s, dtype=torch.bool, device="cuda")
    keep[rows] = False
    assert torch.equal(out[:, keep], out0[:, keep]) and torch.equal(lse[:, :, keep], lse0[:, :, keep])
    assert all(torch.isfinite(g).all() for g in grads)
    dqp, _, dq, _, _ = grads
    assert (dq[:, :, rows] == 0).all() and (dqp[:, :, rows] == 0).all()
    assert torch.equal(dq[:, :, keep], grads0[2][:, :, keep]) and torch.equal(dqp[:, :, keep], grads0[0][:, :, keep])
