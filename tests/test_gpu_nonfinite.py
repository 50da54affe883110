"""Values that are not finite stay with the rows that selected their block: no other row changes by a bit, whatever forward takes
its tile, although the query-tile stationary one multiplies a tile with every block that any of its rows selected."""
import pytest
import torch

from tests.gpu_util import SCALE, bf16_inputs

pytestmark = pytest.mark.gpu


def _poisoned(v, blocks, what):
    bad, zero = v.clone(), v.clone()
    for j in blocks:
        bad[:, :, 128 * j + 7] = what
        zero[:, :, 128 * j + 7] = 0
    return bad, zero


@pytest.mark.parametrize("what", [float("inf"), float("nan")])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("s,kb,blocks", [(1024, 3, [2]), (4224, 20, [1, 17]), (8448, 3, [0, 30])])   # (all tiles, or the first seven)
def test_a_block_that_other_rows_selected(s, kb, blocks, dtype, what):
    from flash_msa_b200 import ops
    cfg = dict(b=1, s=s, hq=4, hkv=2, hp=2, hpkv=1, seed=s)
    qp, kp, q, k, v, _ = bf16_inputs(cfg, dtype=dtype)
    idx = ops.select_blocks(qp, kp, scale=SCALE, num_blocks=s // 128, top_k_blocks=kb)
    rix = ops.build_reverse_index(idx)
    met = torch.stack([(idx == j).any(-1) for j in blocks]).any(0).repeat_interleave(2, 1)

    assert (~met).any() and met.any()

    def run(k, v):
        out, lse, _ = ops.attention_forward(q, k, v, qp, kp, SCALE, rix)
        return out.view(1, s, 4, 128).transpose(1, 2), lse
    bad, zero = _poisoned(v, blocks, what)
    (out, lse), (want, lse0) = run(k, bad), run(k, zero)
    assert torch.isfinite(want).all() and torch.equal(lse, lse0) and torch.equal(out[~met], want[~met])
    assert not torch.isfinite(out[met]).all(-1).any()
    bad, zero = _poisoned(k, blocks, what)
    (out, lse), (want, lse0) = run(bad, v), run(zero, v)
    assert torch.isfinite(want).all() and torch.equal(lse[~met], lse0[~met]) and torch.equal(out[~met], want[~met])


@pytest.mark.parametrize("warmup", [False, True])
def test_documents_that_share_a_tile(warmup):
    """The first document, which ends inside the fourth block, holds the value; the second, whose rows share that tile, does not see it."""
    import flash_msa_b200 as fm
    cfg = dict(b=2, s=1024, hq=4, hkv=2, hp=2, hpkv=1, seed=11)
    qp, kp, q, k, v, _ = bf16_inputs(cfg)
    fn = fm.flash_msa_warmup_varlen_func if warmup else fm.flash_msa_varlen_func

    def run(v):
        with torch.no_grad():
            out, _ = fn(qp, kp, q, k, v, [0, 450, 1024], 8 * 128, SCALE)
        return out.view(2, 1024, 4, 128).transpose(1, 2), torch.zeros(1)
    bad, zero = _poisoned(v, [1], float("inf"))
    out, want = run(bad)[0], run(zero)[0]
    assert torch.equal(out[:, :, :128], want[:, :, :128]) and torch.equal(out[:, :, 450:], want[:, :, 450:])
    assert not torch.isfinite(out[:, :, 256:450]).all(-1).any()


def test_rows_without_their_own_block():
    """Not what a selection gives, but what the index accepts: the first block that a tile visits is not every row's."""
    from flash_msa_b200 import ops
    cfg = dict(b=1, s=512, hq=2, hkv=1, hp=1, hpkv=1, seed=12)
    qp, kp, q, k, v, _ = bf16_inputs(cfg)
    idx = torch.full((1, 1, 512, 2), 4, dtype=torch.int32)
    idx[:, :, 128:384, 0] = 0
    idx[:, :, 200:384, 1] = 1                       # rows 200..255 their own block, and 256.. one before it
    idx[:, :, 384:, 0] = torch.arange(128) % 4      # rows of one tile with four different single blocks
    idx[:, :, 500:, 0] = 4                          # ... and some with none
    rix = ops.build_reverse_index(idx.cuda())
    met = ((idx == 1) | (idx == 3)).any(-1).cuda().repeat_interleave(2, 1)

    def run(v):
        out, lse, _ = ops.attention_forward(q, k, v, qp, kp, SCALE, rix)
        return out.view(1, 512, 2, 128).transpose(1, 2), lse
    bad, zero = _poisoned(v, [1, 3], float("inf"))
    out, lse = run(bad)
    want, lse0 = run(zero)
    assert torch.equal(lse, lse0) and torch.equal(out[~met], want[~met]) and torch.isfinite(want).all()
    none = (idx == 4).all(-1).cuda().repeat_interleave(2, 1)
    assert (out[none] == 0).all()
