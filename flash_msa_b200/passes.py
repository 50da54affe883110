"""Whole forward and backward passes: one C call each (csrc/pipeline.cu) on one workspace.

What depends only on shapes, strides, types and options - the argument block, sizes, layouts - is worked out once and
kept as a plan; a call then fills in pointers.  (Driven stage by stage the host took 0.65 ms for a training pass of
B=1 S=1024 Hq=8, six times what the GPU needs.)"""
from __future__ import annotations

import ctypes
import threading
from ctypes import c_float, c_int32, c_int64, c_void_p

import torch

from . import _lib, ops

_STAGES = ("select_scores", "reverse_index", "attn_fwd", "fwd_combine", "bwd_delta", "attn_bwd", "bwd_combine", "cast")


def _tensor_fields(name):
    return [(name, c_void_p), (name + "_sb", c_int64), (name + "_sh", c_int64), (name + "_ss", c_int64)]


_PROBLEM = list(_lib.FmsaProblem._fields_)
_INPUTS = sum((_tensor_fields(n) for n in ("q", "k", "v", "q_proxy", "k_proxy")), [])
_ORDER = ("q_proxy", "k_proxy", "q", "k", "v")   # of the inputs in a tuple of tensors


class ForwardArgs(ctypes.Structure):
    """Mirror of ``fmsa_forward_args`` with its nested structs laid out flat (same offsets)."""
    _fields_ = _PROBLEM + _INPUTS + [
        ("sinks", c_void_p), ("dense", c_int32), ("with_proxy", c_int32), ("max_partial_bytes", c_int64), ("workspace_bytes", c_int64),
        ("workspace", c_void_p), ("row_ptr", c_void_p), ("col_q", c_void_p), ("edge_pos", c_void_p), ("out", c_void_p),
        ("lse", c_void_p), ("lse_proxy", c_void_p), ("kl_loss", c_void_p), ("status", c_void_p)]


class BackwardArgs(ctypes.Structure):
    """Mirror of ``fmsa_backward_args``, flat."""
    _fields_ = _PROBLEM + _INPUTS + _tensor_fields("d_out") + [
        ("sinks", c_void_p), ("dense", c_int32), ("with_kl", c_int32), ("split_above", c_int32), ("reserved", c_int32),
        ("max_partial_bytes", c_int64), ("workspace_bytes", c_int64), ("workspace", c_void_p), ("row_ptr", c_void_p),
        ("col_q", c_void_p), ("edge_pos", c_void_p), ("out", c_void_p), ("lse", c_void_p), ("lse_proxy", c_void_p),
        ("grad_kl", c_void_p)] + sum((_tensor_fields(n) for n in ("dq", "dk", "dv", "dq_proxy", "dk_proxy")), []) + [
        ("dsinks", c_void_p), ("kl_value", c_void_p), ("status", c_void_p)]


class Marks(ctypes.Structure):
    """Mirror of ``fmsa_marks``."""
    _fields_ = [("events", ctypes.POINTER(c_void_p)), ("stages", ctypes.POINTER(c_int32)), ("capacity", c_int32), ("used", c_int32)]


class _Timing:
    """Events around every stage of one call while `ops.KERNEL_EVENTS` collects them (used by the benchmark)."""
    CAPACITY = 128
    _spare = []

    def __init__(self):
        spare = _Timing._spare
        while len(spare) < self.CAPACITY:
            e = torch.cuda.Event(enable_timing=True)
            e.record()             # creates the CUDA event
            spare.append(e)
        self.handles = (c_void_p * self.CAPACITY)(*(e.cuda_event for e in spare[:self.CAPACITY]))
        self.stages = (c_int32 * self.CAPACITY)()
        self.marks = Marks(ctypes.cast(self.handles, ctypes.POINTER(c_void_p)), ctypes.cast(self.stages, ctypes.POINTER(c_int32)),
                           self.CAPACITY, 0)

    def publish(self):
        n = self.marks.used
        events, _Timing._spare = _Timing._spare[:n], _Timing._spare[n:]
        for i in range(0, n - 1, 2):
            ops.KERNEL_EVENTS.append((_STAGES[self.stages[i]], events[i], events[i + 1]))


def _conforms(stride):
    """Strides that the kernels read in place (see `ops._as_kernel_input`)."""
    return stride[3] == 1 and all(st % 128 == 0 and st > 0 for st in stride[:3])


def _bshd(shape, stride):
    """Whether the tensor is a (B,H,S,D) view of dense (B,S,H,D) storage: its gradient is then written in that layout."""
    b, h, s, d = shape
    return h > 1 and stride == (s * h * d, d, h * d, 1)


class Plan:
    """Everything about a call that shapes, strides, types and options decide."""

    def __init__(self, shapes, layout, dtype, device, top_k_blocks, scale, dense, max_partial_bytes):
        lib = _lib.load()
        hp, hpkv, hkv = (shapes[i][1] for i in (0, 1, 3))
        b, hq, s, d = shapes[2]
        self.dense, self.shape, self.dtype, self.device = dense, (b, hq, s, d), dtype, device
        self.pb = _lib.FmsaProblem(b, s, hq, hkv, hp, hpkv, 1 if dense else int(top_k_blocks), float(scale), ops._dtype_code(dtype), None)
        self.max_partial_bytes = int(max_partial_bytes)
        self.layout = layout
        self.in_place = all(map(_conforms, self.layout))
        self.grad_shapes = [((b, s, sh[1], d), True) if _bshd(sh, st) else (tuple(sh), False) for sh, st in zip(shapes, layout)]
        self.out_shape = (b, s, hq * d)
        pbr = ctypes.byref(self.pb)
        self.forward_bytes = lib.fmsa_forward_workspace_bytes(pbr, int(dense), self.max_partial_bytes)
        self._short_bytes = {}   # see short_documents: by `visible`, of which there are at most S/128
        # saved for the backward, one int32 tensor: row_ptr | col_q | edge_pos | lse | lse_proxy, each from a 64-word boundary
        nb, edges = s // ops.BLOCK_SIZE, 0 if dense else b * hp * s * int(top_k_blocks)
        sizes = [0 if dense else b * hp * nb + 1, edges, edges, b * hq * s, b * hp * s]
        self.at, off = [], 0
        for n in sizes:
            self.at.append(4 * off)
            off += (n + 63) // 64 * 64
        self.saved_words = off
        self.saved_shapes = (*shapes, self.out_shape, (off,))
        self.forward_args = bytes(self._args(ForwardArgs, workspace_bytes=self.forward_bytes))
        self._backward = {}

    def _args(self, kind, **more):
        a = kind(*(getattr(self.pb, f) for f, _ in _PROBLEM), dense=int(self.dense), max_partial_bytes=self.max_partial_bytes, **more)
        for name, stride in zip(_ORDER, self.layout):
            self._strides(a, name, stride)
        return a

    @staticmethod
    def _strides(a, name, stride):
        setattr(a, name + "_sb", stride[0])
        setattr(a, name + "_sh", stride[1])
        setattr(a, name + "_ss", stride[2])

    def backward_template(self, with_kl):
        """(argument block, workspace bytes) of a backward with or without the KL work."""
        got = self._backward.get(with_kl)
        if got is None:
            nbytes = _lib.load().fmsa_backward_workspace_bytes(ctypes.byref(self.pb), int(self.dense), int(with_kl), ops.SPLIT_PARTIALS_ABOVE,
                                                               self.max_partial_bytes)
            a = self._args(BackwardArgs, with_kl=int(with_kl), split_above=ops.SPLIT_PARTIALS_ABOVE, workspace_bytes=nbytes)
            for name, (shape, bshd) in zip(("dq_proxy", "dk_proxy", "dq", "dk", "dv"), self.grad_shapes):
                n1, n2 = shape[1], shape[2]
                self._strides(a, name, (n1 * n2 * 128, 128, n2 * 128) if bshd else (n1 * n2 * 128, n2 * 128, 128))
            got = self._backward[with_kl] = (bytes(a), nbytes)
        return got

    def short_documents(self, visible):
        """Workspace bytes of a forward all of whose tiles go the query-tile stationary way because no tile sees more than
        `visible` blocks; 0 where they do not, or do anyway."""
        got = self._short_bytes.get(visible)
        if got is None:
            lib, pbr, nb = _lib.load(), ctypes.byref(self.pb), self.shape[2] // ops.BLOCK_SIZE
            if self.dense or lib.fmsa_forward_tiles(pbr, 0, visible) < nb or lib.fmsa_forward_tiles(pbr, 0, 0) == nb:
                got = 0
            else:
                got = lib.fmsa_forward_hinted_workspace_bytes(pbr, 0, visible, self.max_partial_bytes)
            self._short_bytes[visible] = got
        return got

    def point(self, a, inputs, as_planned=True):
        """Points the argument block `a` at the inputs as the kernels can read them: in place, or - other strides, or an address
        off the 16-byte grid, which is not part of what a plan knows - copied once into (B,H,S,128) order.  Returns what it points
        at, to be kept until the launch.  The block's strides are those the plan was made for; where the tensors have others
        (`as_planned` False: these inputs; or copies) they are filled in with the addresses."""
        qp, kp, q, k, v = inputs
        pqp, pkp, pq, pk, pv = qp.data_ptr(), kp.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr()
        if as_planned and self.in_place and not (pqp | pkp | pq | pk | pv) & 15:
            a.q_proxy, a.k_proxy, a.q, a.k, a.v = pqp, pkp, pq, pk, pv
            return inputs
        given = [t if _conforms(t.stride()) and t.data_ptr() % 16 == 0 else t.clone(memory_format=torch.contiguous_format) for t in inputs]
        for name, t in zip(_ORDER, given):
            setattr(a, name, t.data_ptr())
            self._strides(a, name, t.stride())
        return given

    def check_unpacked(self, inputs, out, saved):
        """Raises ValueError for tensors that a saved-tensor hook brought back as something else."""
        qp, kp, q, k, v = inputs
        dt, dev = self.dtype, self.device
        if not (qp.dtype is dt and kp.dtype is dt and q.dtype is dt and k.dtype is dt and v.dtype is dt and out.dtype is dt
                and saved.dtype is torch.int32 and qp.device == dev and kp.device == dev and q.device == dev and k.device == dev
                and v.device == dev and out.device == dev and saved.device == dev
                and (qp.shape, kp.shape, q.shape, k.shape, v.shape, out.shape, saved.shape) == self.saved_shapes):
            raise ValueError("the tensors saved for the backward came back with another shape, type or device")


def _whole(t):
    """Contiguous and on the 16-byte grid, as the kernels read `out` and the saved index."""
    return t if t.is_contiguous() and t.data_ptr() % 16 == 0 else t.clone(memory_format=torch.contiguous_format)


_plans = {}
_MAX_PLANS = 256


def plan(inputs, top_k_blocks, scale, dense) -> Plan:
    q = inputs[2]
    shapes, layout = [t.shape for t in inputs], [t.stride() for t in inputs]
    if torch._C._is_tracing():   # sizes are traced tensors then
        shapes = [torch.Size(map(int, sh)) for sh in shapes]
    key = (top_k_blocks, scale, dense, ops.MAX_PARTIAL_BYTES, ops.SPLIT_PARTIALS_ABOVE, q.dtype, q.device, *shapes, *layout)
    p = _plans.get(key)
    if p is None:
        if len(_plans) >= _MAX_PLANS:
            _plans.clear()
        p = _plans[key] = Plan(shapes, layout, q.dtype, q.device, top_k_blocks, scale, dense, ops.MAX_PARTIAL_BYTES)
    return p


def _call(fn, what, args, device):
    timing = _Timing() if ops.KERNEL_EVENTS is not None else None
    launches = c_int32(0)
    _lib.check(fn(ctypes.byref(args), ctypes.byref(timing.marks) if timing else None, ctypes.byref(launches), ops._stream(device)), what)
    ops.LAUNCHES += launches.value
    if timing:
        timing.publish()


def forward(p: Plan, inputs, doc_start, sinks, status_ptr, with_proxy, visible=0):
    """Returns (out [B,S,Hq*128], kl_loss placeholder, saved).  `sinks`: fp32 [Hq] or None.  `with_proxy` False: no backward
    will follow.  `visible`: the most key blocks a query tile can see with `doc_start`, or 0."""
    dev = p.device
    a = ForwardArgs.from_buffer_copy(p.forward_args)
    given = p.point(a, inputs)   # noqa: F841 - copies live until the launch
    out = torch.empty(p.out_shape, dtype=p.dtype, device=dev)
    kl = torch.empty((), dtype=torch.float32, device=dev)
    saved = torch.empty(p.saved_words, dtype=torch.int32, device=dev)
    short = p.short_documents(visible) if visible else 0
    ws = torch.empty(short or p.forward_bytes, dtype=torch.uint8, device=dev)
    if short:
        a.workspace_bytes = short
    base, at = saved.data_ptr(), p.at
    if not p.dense:
        a.row_ptr, a.col_q, a.edge_pos = base + at[0], base + at[1], base + at[2]
    a.lse, a.lse_proxy = base + at[3], base + at[4]
    a.with_proxy = 1 if with_proxy else 0
    a.out, a.kl_loss, a.workspace, a.status = out.data_ptr(), kl.data_ptr(), ws.data_ptr(), status_ptr
    if doc_start is not None:
        a.doc_start = doc_start.data_ptr()
    if sinks is not None:
        a.sinks = sinks.data_ptr()
    lib = _lib.load()
    fn = lib.fmsa_forward
    if short or not with_proxy:
        def fn(args, marks, launches, stream, alone=int(not with_proxy), seen=visible if short else 0):
            return lib.fmsa_forward_hinted(args, alone, seen, marks, launches, stream)
    _call(fn, "fmsa_forward", a, dev)
    return out, kl, saved


def backward(p: Plan, inputs, out, grad_out, saved, grad_kl, kl_value, doc_start, sinks, status_ptr):
    """Returns (dq_proxy, dk_proxy, dq, dk, dv, dsinks) in the type and layout of the forward's inputs; `grad_kl`, `kl_value`:
    fp32 scalars or None.  `inputs`, `out` and `saved` may be other tensors than the forward's (saved-tensor hooks)."""
    dev = p.device
    p.check_unpacked(inputs, out, saved)
    out, saved = _whole(out), _whole(saved)
    hq = p.shape[1]
    if grad_out.dtype != p.dtype:
        grad_out = grad_out.to(p.dtype)
    st = grad_out.stride()
    if grad_out.dim() != 3 or st[2] != 1 or st[0] % 128 or st[1] % 128 or st[0] <= 0 or st[1] <= 0 or grad_out.data_ptr() % 16:
        grad_out = grad_out.reshape(p.out_shape).clone(memory_format=torch.contiguous_format)
        st = grad_out.stride()
    template, nbytes = p.backward_template(grad_kl is not None)
    a = BackwardArgs.from_buffer_copy(template)
    given = p.point(a, inputs, [t.stride() for t in inputs] == p.layout)   # noqa: F841 - copies live until the launch
    ws = torch.empty(nbytes, dtype=torch.uint8, device=dev)
    grads = [torch.empty(shape, dtype=p.dtype, device=dev) for shape, _ in p.grad_shapes]
    a.d_out, a.d_out_sb, a.d_out_sh, a.d_out_ss = grad_out.data_ptr(), st[0], 128, st[1]
    a.dq_proxy, a.dk_proxy, a.dq, a.dk, a.dv = (g.data_ptr() for g in grads)
    base, at = saved.data_ptr(), p.at
    if not p.dense:
        a.row_ptr, a.col_q, a.edge_pos = base + at[0], base + at[1], base + at[2]
    a.lse, a.lse_proxy = base + at[3], base + at[4]
    a.out, a.workspace, a.status = out.data_ptr(), ws.data_ptr(), status_ptr
    if grad_kl is not None:
        if grad_kl.dtype != torch.float32 or grad_kl.device != dev:
            grad_kl = grad_kl.to(device=dev, dtype=torch.float32)
        a.grad_kl = grad_kl.data_ptr()
        if kl_value is not None:
            a.kl_value = kl_value.data_ptr()
    if doc_start is not None:
        a.doc_start = doc_start.data_ptr()
    dsinks = None
    if sinks is not None:
        dsinks = torch.empty(hq, dtype=torch.float32, device=dev)
        a.sinks, a.dsinks = sinks.data_ptr(), dsinks.data_ptr()
    _call(_lib.load().fmsa_backward, "fmsa_backward", a, dev)
    return [g.transpose(1, 2) if bshd else g for g, (_, bshd) in zip(grads, p.grad_shapes)] + [dsinks]


class StatusBoard:
    """Status words of the calls of this process, in pinned host memory that the kernels write directly (only ever when
    something is wrong), so that a call needs no word of its own, no copy and no event.  There is one word for each of a few
    kinds of call, shared by all threads, streams and devices: it says what kind of call met trouble, not whose it was, and the
    RuntimeError is raised by whichever call of the library comes next, or by `drain`."""
    KINDS = ("flash_msa_func forward", "flash_msa_func backward", "flash_msa_warmup_func forward", "flash_msa_warmup_func backward")

    def __init__(self):
        self._words = None
        self._devices = set()
        self._lock = threading.Lock()

    def pointer(self, kind: int, device) -> int:
        if self._words is None:
            with self._lock:   # of several first calls one makes the words; kernels hold on to their address
                if self._words is None:
                    self._keep = torch.zeros(16, dtype=torch.int32).pin_memory()
                    self._words = (c_int32 * 16).from_address(self._keep.data_ptr())
        self._devices.add(device)
        self.poll()
        return ctypes.addressof(self._words) + 4 * kind

    def poll(self) -> None:
        if self._words is not None and any(self._words):
            for i, what in enumerate(self.KINDS):
                code = self._words[i]
                if code:
                    self._words[i] = 0
                    raise RuntimeError(f"{what} (reported late): {ops._STATUS_NAMES.get(code, code)}")

    def drain(self) -> None:
        for device in list(self._devices):
            torch.cuda.synchronize(device)
        self.poll()


status_board = StatusBoard()
