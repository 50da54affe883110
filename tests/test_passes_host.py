"""Host side of the whole-pass calls, without a GPU: what an argument block says about the tensors whose pointers it holds.
The native call is replaced by a recorder, so that nothing is launched."""
import ctypes
import threading
import time

import numpy as np
import pytest
import torch
from torch.autograd import forward_ad

from flash_msa_b200 import passes
from oracle import msa_oracle as O

B, H, HKV, S = 2, 4, 2, 256
NAMES = ("q_proxy", "k_proxy", "q", "k", "v")


def _dense(h, fill):
    return torch.arange(B * h * S * 128, dtype=torch.float32).remainder_(61).add_(fill).to(torch.bfloat16).view(B, h, S, 128)


def _strided(t, kind):
    """`t`'s values in another layout."""
    b, h, s, d = t.shape
    if kind == "dense":
        return t.clone()
    if kind == "bshd":
        return t.transpose(1, 2).contiguous().transpose(1, 2)
    if kind in ("packed", "packed_shifted"):      # some heads of a (B,S,2H,128) buffer, which may begin one element late
        shift = 1 if kind == "packed_shifted" else 0
        buf = torch.zeros(b * s * 2 * h * d + 8, dtype=t.dtype)
        view = buf[shift:shift + b * s * 2 * h * d].view(b, s, 2 * h, d)[:, :, :h].transpose(1, 2)
        return view.copy_(t)
    if kind == "shifted":                          # dense, but not on a 16-byte boundary
        return torch.empty(t.numel() + 8, dtype=t.dtype)[3:3 + t.numel()].view(t.shape).copy_(t)
    if kind == "wide":                             # rows 136 elements apart
        return torch.zeros(b, h, s, d + 8, dtype=t.dtype)[..., :d].copy_(t)
    if kind == "expanded":                         # every head the same memory
        return t[:, :1].clone().expand(b, h, s, d)
    raise ValueError(kind)


KINDS = ["dense", "bshd", "packed", "packed_shifted", "shifted", "wide", "expanded"]


class _Recorder:
    """Stands in for the native call; `given` are the tensors that `Plan.point` points it at."""

    def __init__(self, monkeypatch):
        self.blocks, self.given = [], []
        point = passes.Plan.point

        def watch(plan, *args):
            self.given.append(list(point(plan, *args)))
            return self.given[-1]
        monkeypatch.setattr(passes.Plan, "point", watch)
        monkeypatch.setattr(passes, "_call", lambda fn, what, a, device: self.blocks.append(type(a).from_buffer_copy(a)))

    def check(self, block, given, inputs):
        for name, t, asked in zip(NAMES, given, inputs):
            assert getattr(block, name) == t.data_ptr() and t.data_ptr() % 16 == 0, name
            strides = tuple(getattr(block, f"{name}_{x}") for x in ("sb", "sh", "ss"))
            assert strides + (1,) == t.stride(), name
            assert all(st > 0 and st % 128 == 0 for st in strides), name
            assert torch.equal(t, asked), name


@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("kind", KINDS)
def test_strides_in_the_argument_block_are_those_of_the_tensors(monkeypatch, kind, dense):
    """An input that cannot be read in place is copied, and then the copy's strides are what the kernels get: also when its
    strides alone would do and only its address does not (the clone of a slice does not have the slice's strides)."""
    rec = _Recorder(monkeypatch)
    inputs = tuple(_strided(_dense(h, i), kind) for i, h in enumerate((2, 1, H, HKV, HKV)))
    plan = passes.plan(inputs, 0 if dense else 1, 0.1, dense)
    out, _, saved = passes.forward(plan, inputs, None, None, 0, True)
    passes.backward(plan, inputs, out, torch.zeros_like(out), saved, torch.ones(()), None, None, None, 0)
    for block, given in zip(rec.blocks, rec.given):
        rec.check(block, given, inputs)
    # the same shapes and strides on a 16-byte boundary, and then off it again: nothing is remembered of the address
    again = [_strided(t.contiguous(), "packed") if kind == "packed_shifted" else t for t in inputs]
    for tensors in (again, inputs):
        passes.forward(passes.plan(tensors, 0 if dense else 1, 0.1, dense), tensors, None, None, 0, True)
        rec.check(rec.blocks[-1], rec.given[-1], tensors)


@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("first", ["dense", "bshd", "packed"])
@pytest.mark.parametrize("then", [kind for kind in KINDS if kind != "expanded"])   # (an unpacked tensor has the packed one's values)
def test_backward_takes_the_strides_of_what_it_is_given(monkeypatch, first, then, dense):
    """Saved-tensor hooks hand the backward other tensors than the forward had: `torch.autograd.graph.save_on_cpu` brings
    every input back contiguous, whatever it was, a hook that packs them into one buffer brings back slices."""
    rec = _Recorder(monkeypatch)
    values = [_dense(h, i) for i, h in enumerate((2, 1, H, HKV, HKV))]
    inputs = tuple(_strided(t, first) for t in values)
    plan = passes.plan(inputs, 0 if dense else 1, 0.1, dense)
    out, _, saved = passes.forward(plan, inputs, None, None, 0, True)
    unpacked = tuple(_strided(t, then) for t in values)
    odd = torch.empty(out.numel() + 8, dtype=out.dtype)[1:1 + out.numel()].view(out.shape)
    grads = passes.backward(plan, unpacked, odd, torch.zeros_like(out), saved, torch.ones(()), None, None, None, 0)
    rec.check(rec.blocks[1], rec.given[1], values)
    assert rec.blocks[1].out % 16 == 0
    # the gradients keep the layout of the forward's inputs, which are the leaves
    for name, g, t in zip(NAMES, grads, inputs):
        assert getattr(rec.blocks[1], "d" + name) == g.data_ptr() and g.shape == t.shape
        assert tuple(getattr(rec.blocks[1], f"d{name}_{x}") for x in ("sb", "sh", "ss")) + (1,) == g.stride()


@pytest.mark.parametrize("odd", [{"dtype": torch.float16}, {"shape": True}, {"device": "meta"}])
@pytest.mark.parametrize("which", range(7))
def test_backward_refuses_tensors_of_another_kind(monkeypatch, which, odd):
    """What comes back from a hook with another type, shape or device is refused instead of read."""
    monkeypatch.setattr(passes, "_call", lambda fn, what, a, device: None)
    inputs = [_dense(h, i) for i, h in enumerate((2, 1, H, HKV, HKV))]
    plan = passes.plan(inputs, 1, 0.1, False)
    out, _, saved = passes.forward(plan, inputs, None, None, 0, True)
    ts = inputs + [out, saved]
    ts[which] = ts[which][..., :64] if "shape" in odd else ts[which].to(**odd)
    with pytest.raises(ValueError, match="backward"):
        passes.backward(plan, ts[:5], ts[5], torch.zeros_like(out), ts[6], None, None, None, None, 0)


class _SaysCuda(torch.Tensor):
    """A CPU tensor that reports `where` as its device (no launch is reached with it)."""
    where = torch.device("cuda", 0)
    device = property(lambda self: self.where)


@pytest.mark.parametrize("warmup", [False, True])
@pytest.mark.parametrize("odd", [0, 1, 3, 4])
@pytest.mark.parametrize("where", ["cpu", "cuda:1"])
def test_inputs_on_another_device_than_q_are_refused(monkeypatch, where, odd, warmup):
    import flash_msa_b200 as fm
    monkeypatch.setattr(passes, "forward", lambda *a, **k: pytest.fail("a call with tensors on two devices went through"))
    inputs = [_dense(h, i).as_subclass(_SaysCuda) for i, h in enumerate((2, 1, H, HKV, HKV))]
    inputs[odd].where = torch.device(where)
    fn = fm.flash_msa_warmup_func if warmup else fm.flash_msa_func
    with pytest.raises(ValueError, match="device"):
        fn(*inputs, 128, 0.1)
    # (a q that is not on a GPU keeps its own error)
    with pytest.raises(RuntimeError, match="CUDA"):
        fn(*(_dense(h, i) for i, h in enumerate((2, 1, H, HKV, HKV))), 128, 0.1)


@pytest.fixture
def on_the_host(monkeypatch):
    """The public functions on CPU tensors, with a forward that copies q's storage to `out` behind torch's back."""
    from flash_msa_b200 import api

    def forward(p, inputs, doc_start, sinks, status_ptr, with_proxy):
        out = torch.empty(p.out_shape, dtype=p.dtype)
        ctypes.memmove(out.data_ptr(), inputs[2].data_ptr(), 2 * out.numel())
        if doc_start is not None:
            ctypes.memmove(out.data_ptr(), doc_start.data_ptr(), 4 * doc_start.numel())
        return out, torch.zeros(()), torch.zeros(p.saved_words, dtype=torch.int32)
    monkeypatch.setattr(passes, "forward", forward)
    monkeypatch.setattr(passes.status_board, "pointer", lambda kind, device: 0)
    monkeypatch.setattr(api, "_require_cuda", lambda *a: None)
    return api


@pytest.mark.filterwarnings("ignore::torch.jit.TracerWarning")
@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("warmup", [False, True])
def test_a_trace_calls_the_library(on_the_host, grad, warmup):
    """A traced function runs the call again on what it is given, also with other sizes, and refuses what the call refuses."""
    import flash_msa_b200 as fm
    fn = fm.flash_msa_warmup_func if warmup else fm.flash_msa_func

    def values(seed, b=B):
        g = torch.Generator().manual_seed(seed)
        return tuple(torch.randn(b, h, S, 128, generator=g).to(torch.bfloat16) for h in (2, 1, H, HKV, HKV))
    with torch.set_grad_enabled(grad):
        first = tuple(t.requires_grad_(grad) for t in values(1))
        traced = torch.jit.trace(lambda *ts: fn(*ts, 128, 0.1), first, check_trace=False)
        for ts in (values(2), values(3, b=1)):
            out, _ = traced(*ts)
            assert torch.equal(out.detach().flatten(), ts[2].flatten())
        with pytest.raises((ValueError, RuntimeError), match="divisible by 128"):
            traced(*(t[:, :, :200] for t in values(4)))


@pytest.mark.filterwarnings("ignore::torch.jit.TracerWarning")
def test_a_trace_keeps_document_boundaries(on_the_host):
    import flash_msa_b200 as fm
    ts = tuple(_dense(h, i) for i, h in enumerate((2, 1, H, HKV, HKV)))
    with torch.no_grad():
        traced = torch.jit.trace(lambda *a: fm.flash_msa_varlen_func(*a, [0, 100, S], 128, 0.1), ts, check_trace=False)
        out, _ = traced(*ts)
    doc_start = out.flatten()[:2 * B * S].view(torch.int32).view(B, S)
    assert torch.equal(doc_start, torch.tensor([0] * 100 + [100] * (S - 100), dtype=torch.int32).expand(B, S))


@pytest.mark.parametrize("warmup", [False, True])
def test_transforms_without_a_rule_are_refused(monkeypatch, warmup):
    """Tangents would be lost without a word, and batched tensors have no memory of their own."""
    import flash_msa_b200 as fm
    from flash_msa_b200 import api
    launched = []
    monkeypatch.setattr(passes, "_call", lambda *a: launched.append(a))
    monkeypatch.setattr(passes.status_board, "pointer", lambda kind, device: 0)
    monkeypatch.setattr(api, "_require_cuda", lambda *a: None)
    fn = fm.flash_msa_warmup_func if warmup else fm.flash_msa_func
    inputs = [_dense(h, i) for i, h in enumerate((2, 1, H, HKV, HKV))]
    for grad in (False, True):
        with torch.set_grad_enabled(grad), forward_ad.dual_level():
            q = forward_ad.make_dual(inputs[2], torch.ones_like(inputs[2]))
            with pytest.raises(NotImplementedError, match="jvp"):
                fn(*inputs[:2], q, *inputs[3:], 128, 0.1)
        launched.clear()   # (the autograd function runs its forward before it looks for a rule)
        with torch.set_grad_enabled(grad), pytest.raises(RuntimeError):
            torch.func.vmap(lambda *ts: fn(*ts, 128, 0.1))(*(t.unsqueeze(0) for t in inputs))
        assert not launched


def test_first_calls_of_several_threads_share_one_status_board(monkeypatch):
    """Pinning takes a while, and every thread that makes its first call meanwhile must end up with the same words."""
    pinned = []

    def pin(t):
        time.sleep(0.05)
        pinned.append(t)
        return t
    monkeypatch.setattr(torch.Tensor, "pin_memory", pin)
    board, start, got = passes.StatusBoard(), threading.Barrier(8), []

    def call(i):
        start.wait()
        got.append(board.pointer(i % 4, torch.device("cuda", 0)) - 4 * (i % 4))
    threads = [threading.Thread(target=call, args=(i,)) for i in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(pinned) == 1 and got == [pinned[0].data_ptr()] * 8
    ctypes.c_int32.from_address(got[0] + 4).value = 2
    with pytest.raises(RuntimeError, match="flash_msa_func backward.*out-of-range index"):
        board.pointer(0, torch.device("cuda", 0))
    assert board.pointer(0, torch.device("cuda", 0)) == got[0]     # raised once


@pytest.mark.parametrize("form", ["list", "tuple", "range", "int32", "bf16", "scalars", "numpy", "per_batch"])
def test_forms_of_document_boundaries(form):
    """Whatever torch.as_tensor takes is taken, from host memory as well."""
    from flash_msa_b200 import ops
    cu = [0, 64, 192, 256]
    given = {"list": cu, "tuple": tuple(cu), "range": range(0, 257, 64), "int32": torch.tensor(cu, dtype=torch.int32),
             "bf16": torch.tensor(cu).to(torch.bfloat16), "scalars": [torch.tensor(x) for x in cu],
             "numpy": np.array(cu, dtype=np.int16), "per_batch": [cu, [0, 0, 1, 256]]}[form]
    got = ops.doc_start_from_cu_seqlens(given, 2, 256, torch.device("cpu"))
    assert torch.equal(got, O.doc_start_from_cu_seqlens(list(given) if form == "range" else given if form == "per_batch" else cu, 256, 2))
    for bad in ([0, 5, 3, 256], [1, 256], [0, 255], [0], [[0, 256]] * 3):
        with pytest.raises(ValueError):
            ops.doc_start_from_cu_seqlens(bad, 2, 256, torch.device("cpu"))


@pytest.mark.parametrize("dense", [False, True])
def test_short_documents_are_asked_for_once(monkeypatch, dense):
    """What a plan's forward needs for documents that span so many blocks depends on nothing else: the library is asked once, and
    the answers are those that it gives."""
    from flash_msa_b200 import _lib
    s, kb = 128 * 40, 3
    inputs = [torch.empty(1, h, s, 128, dtype=torch.bfloat16) for h in (2, 1, 8, 2, 2)]
    plan = passes.Plan([t.shape for t in inputs], [t.stride() for t in inputs], torch.bfloat16, inputs[0].device, kb, 0.1, dense, 1 << 32)
    lib, pb, asked = _lib.load(), ctypes.byref(plan.pb), []

    class Counting:
        def __getattr__(self, name):
            asked.append(name)
            return getattr(lib, name)
    monkeypatch.setattr(_lib, "load", Counting)
    counts = []
    for _ in range(2):
        for visible in range(1, 41):
            all_tiles = not dense and lib.fmsa_forward_tiles(pb, 0, visible) == 40
            assert all_tiles == (not dense and visible <= 5 * kb // 2)
            assert plan.short_documents(visible) == (lib.fmsa_forward_hinted_workspace_bytes(pb, 0, visible, 1 << 32) if all_tiles else 0)
        counts.append(len(asked))
    assert counts[0] == counts[1]
