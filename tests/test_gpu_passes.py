"""The whole-pass entry points where they branch: softmax sinks with one and several groups of heads in the log-sum-exp
kernel, inputs that have to be copied first, a forward without a backward, document boundaries from host and device
memory, the status words in host memory."""
import pytest
import torch

from oracle import msa_oracle as O
from tests.gpu_util import SCALE, bf16_inputs, forward_tiles, kernel_selection, max_err, yardstick_check

pytestmark = pytest.mark.gpu
NAMES = ["dq_proxy", "dk_proxy", "dq", "dk", "dv"]


@pytest.mark.parametrize("mpp,s,kb", [(1, 384, 2), (8, 384, 2), (9, 384, 2), (12, 384, 2), (1, 5120, 1), (8, 3072, 1), (9, 3072, 2), (12, 3072, 1)])
def test_sinks_over_groups_of_heads(mpp, s, kb):
    """The query-tile stationary forward alone (384), whose log-sum-exps take the sinks in a kernel of their own, and with the key-block
    stationary one behind it, whose combine takes them."""
    import flash_msa_b200 as fm
    cfg = dict(b=2, s=s, hq=2 * mpp, hkv=2, hp=2, hpkv=1, kb=kb, seed=80 + mpp)
    qp, kp, q, k, v, do = bf16_inputs(cfg)
    assert forward_tiles((qp, kp, q, k, v), kb) == (3 if s == 384 else 5 * kb // 2)
    sinks = (torch.randn(cfg["hq"], generator=torch.Generator().manual_seed(mpp)) + 1.0).cuda().requires_grad_(True)
    leaves = [t.detach().requires_grad_(True) for t in (qp, kp, q, k, v)]
    out, kl = fm.flash_msa_func(*leaves, cfg["kb"] * 128, SCALE, sinks=sinks)
    torch.autograd.backward([out, kl], [do, torch.ones((), device="cuda")])
    idx = kernel_selection(qp, kp, cfg["kb"])
    args = (qp, kp, q, k, v, cfg["kb"] * 128, SCALE, do, 1.0)
    r32 = O.sparse_forward_backward(*args, block_indices=idx, sinks=sinks.detach())
    r16 = O.sparse_forward_backward(*args, block_indices=idx, sinks=sinks.detach(), dtype=torch.bfloat16)
    yardstick_check("out", out, r32["out"], r16["out"], 2e-3)
    for n, leaf in zip(NAMES, leaves):
        yardstick_check(n, leaf.grad, r32[n], r16[n], 2e-3 * r32[n].abs().max().item())
    # (a sum over all rows of a head of exp(sink - lse) * delta, delta formed from the 16-bit output)
    assert max_err(sinks.grad, r32["dsinks"]) <= 1e-2 * max(1.0, r32["dsinks"].abs().max().item())


@pytest.mark.parametrize("warmup", [False, True])
def test_copied_inputs_and_forward_alone(warmup):
    """Strides the kernels cannot read in place (rows 136 elements apart) and a pass without gradients give the plain result."""
    import flash_msa_b200 as fm
    cfg = dict(b=2, s=512, hq=6, hkv=2, hp=2, hpkv=2, kb=3, seed=90)
    *inputs, do = bf16_inputs(cfg)
    fn = fm.flash_msa_warmup_func if warmup else fm.flash_msa_func
    res = []
    for widen in (False, True):
        base = [torch.nn.functional.pad(t, (0, 8))[..., :128] if widen else t for t in inputs]
        assert base[0].stride(2) == (136 if widen else 128)
        leaves = [t.detach().requires_grad_(True) for t in base]
        out, kl = fn(*leaves, 384, SCALE)
        torch.autograd.backward([out, kl], [do, torch.ones((), device="cuda")])
        with torch.no_grad():
            alone, kl0 = fn(*base, 384, SCALE)
        assert torch.equal(alone, out) and kl0.item() == 0.0 and not alone.requires_grad
        res.append([out] + [t.grad for t in leaves])
    for n, a, b in zip(["out"] + NAMES, *res):
        assert max_err(a, b) <= (0.0 if n in ("out", "dq", "dq_proxy") else 2 ** -7 * a.float().abs().max().item()), n


@pytest.mark.parametrize("warmup", [False, True])
def test_slices_off_the_16_byte_grid(warmup):
    """Heads of a wider buffer that begins one element late: strides the kernels could read, an address they cannot, so every
    input is copied and the copy's strides count (tests/test_passes_host.py).  The plain result, bit for bit where sums have a
    fixed order."""
    import flash_msa_b200 as fm
    cfg = dict(b=2, s=512, hq=6, hkv=2, hp=2, hpkv=2, kb=3, seed=91)
    *inputs, do = bf16_inputs(cfg)
    fn = fm.flash_msa_warmup_func if warmup else fm.flash_msa_func

    def late(t):
        b, h, s, d = t.shape
        view = torch.zeros(b * s * 2 * h * d + 8, dtype=t.dtype, device=t.device)[1:-7].view(b, s, 2 * h, d)[:, :, :h].transpose(1, 2)
        assert view.data_ptr() % 16 == 2 and view.stride() == (2 * s * h * d, d, 2 * h * d, 1)
        return view.copy_(t)
    res = []
    for base in (inputs, [late(t) for t in inputs]):
        leaves = [t.detach().requires_grad_(True) for t in base]
        out, kl = fn(*leaves, 384, SCALE)
        torch.autograd.backward([out, kl], [do, torch.ones((), device="cuda")])
        res.append([out] + [t.grad for t in leaves])
    for n, a, b in zip(["out"] + NAMES, *res):
        assert max_err(a, b) <= (0.0 if n in ("out", "dq", "dq_proxy") else 2 ** -7 * a.float().abs().max().item()), n


@pytest.mark.parametrize("warmup", [False, True])
def test_saved_tensors_kept_on_the_host(warmup):
    """`save_on_cpu` brings the inputs back contiguous although they were views of (B,S,H,D) storage."""
    import flash_msa_b200 as fm
    cfg = dict(b=2, s=512, hq=6, hkv=2, hp=2, hpkv=2, kb=3, seed=92)
    *inputs, do = bf16_inputs(cfg, layout="bshd")
    fn = fm.flash_msa_warmup_func if warmup else fm.flash_msa_func
    res = []
    for offload in (False, True):
        leaves = [t.detach().requires_grad_(True) for t in inputs]
        if offload:
            with torch.autograd.graph.save_on_cpu():
                out, kl = fn(*leaves, 384, SCALE)
        else:
            out, kl = fn(*leaves, 384, SCALE)
        torch.autograd.backward([out, kl], [do, torch.ones((), device="cuda")])
        res.append([t.grad for t in leaves])
    for n, a, b in zip(NAMES, *res):
        assert a.stride() == b.stride()
        assert max_err(a, b) <= (0.0 if n in ("dq", "dq_proxy") else 2 ** -7 * a.float().abs().max().item()), n


@pytest.mark.parametrize("dense,kl,cap,cu", [(False, True, None, None), (False, False, 1, None), (True, True, 1, None),
                                             (False, True, None, [0, 100, 640]), (True, False, None, [0, 100, 640])])
def test_single_stages_agree_with_whole_passes(monkeypatch, dense, kl, cap, cu):
    """The stage entry points, which other bindings call one by one, against the whole-pass calls that drive the same kernels:
    bit for bit where sums have a fixed order, also over several passes."""
    import flash_msa_b200 as fm
    from flash_msa_b200 import ops
    if cap:
        monkeypatch.setattr(ops, "MAX_PARTIAL_BYTES", cap)
    cfg = dict(b=2, s=640, hq=12, hkv=2, hp=4, hpkv=2, kb=2, seed=93)
    qp, kp, q, k, v, do = bf16_inputs(cfg)
    gk = torch.ones((), device="cuda") if kl else None
    leaves = [t.detach().requires_grad_(True) for t in (qp, kp, q, k, v)]
    fn = {(False, False): fm.flash_msa_func, (True, False): fm.flash_msa_warmup_func, (False, True): fm.flash_msa_varlen_func,
          (True, True): fm.flash_msa_warmup_varlen_func}[dense, cu is not None]
    out, kl_loss = fn(*leaves, *([] if cu is None else [cu]), cfg["kb"] * 128, SCALE)
    torch.autograd.backward([out, kl_loss] if kl else [out], [do, gk] if kl else [do])
    ds = None if cu is None else ops.doc_start_from_cu_seqlens(cu, cfg["b"], cfg["s"], qp.device)
    rix = None if dense else ops.build_reverse_index(ops.select_blocks_fused(qp, kp, SCALE, cfg["kb"], doc_start=ds))
    out2, lse, lse_p = ops.attention_forward(q, k, v, qp, kp, SCALE, rix, dense=dense, doc_start=ds)
    grads = ops.attention_backward(q, k, v, qp, kp, out2, do, lse, lse_p, SCALE, rix, gk, dense=dense, doc_start=ds)
    assert torch.equal(out, out2)
    for n, leaf, b in zip(NAMES, leaves, grads):
        a = torch.zeros_like(b) if leaf.grad is None else leaf.grad
        assert max_err(a, b) <= (0.0 if n in ("dq", "dq_proxy") else 2 ** -7 * b.float().abs().max().item()), n


@pytest.mark.parametrize("cu", [[0, 512], [0, 0, 1, 130, 130, 511, 512, 512], [[0, 7, 512], [0, 512, 512]], list(range(0, 513)) + [512] * 500])
def test_document_boundaries_from_the_host(cu):
    """Short lists travel as a kernel parameter, long ones and device tensors take the other way: the same array."""
    from flash_msa_b200 import ops
    dev = torch.device("cuda", 0)
    got = ops.doc_start_from_cu_seqlens(cu, 2, 512, dev)
    assert torch.equal(got, ops.doc_start_from_cu_seqlens(torch.tensor(cu, device=dev), 2, 512, dev))
    assert torch.equal(got.cpu(), O.doc_start_from_cu_seqlens(cu, 512, 2))
    for bad in ([0, 5, 3, 512], [1, 512], [0, 511]):
        with pytest.raises(ValueError):
            ops.doc_start_from_cu_seqlens(bad, 2, 512, dev)


def test_status_words_in_host_memory():
    """A kernel whose bounded wait ran out writes its status word into pinned host memory; the next look raises once."""
    from flash_msa_b200 import _lib, passes
    board = passes.StatusBoard()
    dev = torch.device("cuda", 0)
    g = torch.Generator(device="cpu").manual_seed(14)
    src, b = (torch.randn(n, 128, generator=g).to(torch.bfloat16).cuda() for n in (256, 128))
    rows = torch.arange(128, dtype=torch.int32).cuda()
    d = torch.zeros(2, 128, 128, device=dev)
    part = torch.zeros(128, 2, 128, dtype=torch.bfloat16, device=dev)
    for withhold in (0, 1):
        _lib.check(_lib.load().fmsa_pipeline_selftest(src.data_ptr(), 256, rows.data_ptr(), b.data_ptr(), d[0].data_ptr(), d[1].data_ptr(),
                                                      part.data_ptr(), withhold, 2_000_000, board.pointer(1, dev), None), "selftest")
        if not withhold:
            board.drain()
    with pytest.raises(RuntimeError, match="flash_msa_func backward.*timed out"):
        board.drain()
    board.drain()
