"""Two planes of backward partial rows (values and rounding remainders), which only rows with many selected blocks take by
themselves, at small sizes where the ends of the reverse-index rows fall anywhere in a tile: both halves of a tile, 32-query
steps and rows of one query; bf16 and fp16, packed documents, with and without KL work."""
import pytest
import torch

from oracle import msa_oracle as O
from tests.gpu_util import SCALE, bf16_inputs, kernel_selection, max_err, yardstick_check

pytestmark = pytest.mark.gpu
NAMES = ["dq_proxy", "dk_proxy", "dq", "dk", "dv"]


def _grads(fm, inputs, do, kb, kl_work, cu):
    leaves = [t.detach().requires_grad_(True) for t in inputs]
    out, kl = fm.flash_msa_func(*leaves, kb * 128, SCALE) if cu is None else fm.flash_msa_varlen_func(*leaves, cu, kb * 128, SCALE)
    torch.autograd.backward([out, kl] if kl_work else [out], [do, torch.ones((), device="cuda")] if kl_work else [do])
    return [t.grad for t in leaves]


@pytest.mark.parametrize("s,mpp,kb,dtype,kl_work", [(128, 1, 1, "bf16", True), (640, 3, 2, "bf16", True), (640, 3, 2, "bf16", False),
                                                    (1152, 1, 3, "fp16", True), (896, 2, 7, "fp16", False)])
def test_two_planes_at_ragged_rows(monkeypatch, s, mpp, kb, dtype, kl_work):
    import flash_msa_b200 as fm
    from flash_msa_b200 import ops
    cfg = dict(b=2, s=s, hq=2 * mpp, hkv=1, hp=2, hpkv=1, kb=kb, seed=31 + s)
    t16 = torch.bfloat16 if dtype == "bf16" else torch.float16
    *inputs, do = [t.to(t16) for t in bf16_inputs(cfg)]
    monkeypatch.setattr(ops, "SPLIT_PARTIALS_ABOVE", 0)
    two = _grads(fm, inputs, do, kb, kl_work, None)
    packed = _grads(fm, inputs, do, kb, kl_work, [0, s])   # the kernels with document masking, nothing masked
    idx = kernel_selection(inputs[0], inputs[1], kb)
    args = (*inputs, kb * 128, SCALE, do, 1.0 if kl_work else None)
    r32 = O.sparse_forward_backward(*args, block_indices=idx)
    r16 = O.sparse_forward_backward(*args, block_indices=idx, dtype=t16)
    for n, a, p in zip(NAMES, two, packed):
        if kl_work or "proxy" not in n:
            yardstick_check(n, a, r32[n], r16[n], 2e-3 * r32[n].abs().max().item())
        assert max_err(a, p) <= (0.0 if n in ("dq", "dq_proxy") else 2 ** -7 * a.float().abs().max().item()), n
