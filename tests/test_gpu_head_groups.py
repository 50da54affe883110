"""The combine kernels beyond eight main heads per proxy head: blocks take groups of at most six heads, whose pieces of the
partial-row records start inside a record, and more than nine statistics per edge need two groups of the log-sum-exp
kernel.  Sizes at the edges of the groups (9 = 5 + 4, 13 = 5 + 5 + 3, 18 = 6 + 6 + 6), one and two planes of partial rows."""
import pytest
import torch

from oracle import msa_oracle as O
from tests.gpu_util import SCALE, bf16_inputs, forward_tiles, kernel_selection, yardstick_check

pytestmark = pytest.mark.gpu
NAMES = ["dq_proxy", "dk_proxy", "dq", "dk", "dv"]


@pytest.mark.parametrize("mpp,s,kb", [(9, 640, 2), (13, 640, 3), (18, 640, 2), (9, 4352, 33),
                                      (9, 4096, 1), (13, 3072, 1), (18, 3072, 1)])   # the last three: the forward's combine too
def test_groups_of_main_heads(mpp, s, kb):
    import flash_msa_b200 as fm
    cfg = dict(b=1, s=s, hq=mpp, hkv=1, hp=1, hpkv=1, kb=kb, seed=60 + mpp)
    qp, kp, q, k, v, do = bf16_inputs(cfg)
    assert forward_tiles((qp, kp, q, k, v), kb) == (s // 128 if s in (640, 4352) else 2)
    leaves = [t.detach().requires_grad_(True) for t in (qp, kp, q, k, v)]
    out, kl = fm.flash_msa_func(*leaves, kb * 128, SCALE)
    torch.autograd.backward([out, kl], [do, torch.ones((), device="cuda")])
    idx = kernel_selection(qp, kp, kb)
    r32 = O.sparse_forward_backward(qp, kp, q, k, v, kb * 128, SCALE, do, 1.0, block_indices=idx)
    r16 = O.sparse_forward_backward(qp, kp, q, k, v, kb * 128, SCALE, do, 1.0, block_indices=idx, dtype=torch.bfloat16)
    yardstick_check("out", out, r32["out"], r16["out"], 1e-3)
    for n, leaf in zip(NAMES, leaves):
        yardstick_check(n, leaf.grad, r32[n], r16[n], 2e-3 * r32[n].abs().max().item())
