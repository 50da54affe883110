"""Autograd boundary: the reference's public functions with the same arguments, layouts, return
values and error behaviour (flash_msa/flash_msa.py:19-64, 129-278;
flash_msa/warmup/flash_msa_warmup.py:6-106), on top of the sm_100a kernels."""
from __future__ import annotations

import torch
from torch.autograd import forward_ad

from . import ops, passes

BLOCK_SIZE = 128
MAX_TOP_K_BLOCKS = 128

# The device status word of every call (a bounded wait that ran out, a bad index in metadata) is looked at
# without synchronising: the kernels write it to pinned host memory, and the next call of the library raises
# RuntimeError; `check_pending_status()` waits for everything queued so far.
# DEBUG_CHECK_STATUS = True reads a word of the call's own right after every call instead (synchronises; for debugging).
DEBUG_CHECK_STATUS = False


def _validate_inputs(q_proxy, k_proxy, q, k, v, top_k, sparse: bool):
    if q_proxy.ndim != 4 or k_proxy.ndim != 4 or q.ndim != 4 or k.ndim != 4 or v.ndim != 4:
        raise ValueError("all attention tensors must have shape (B, H, S, D)")
    b, n_proxy_heads, s, head_dim = q_proxy.shape
    bk, n_proxy_kv_heads, sk, dk = k_proxy.shape
    bq, n_heads, sq, dq = q.shape
    bm, n_kv_heads, sm, dm = k.shape
    bv, n_v_heads, sv, dv = v.shape
    if not (b == bk == bq == bm == bv and s == sk == sq == sm == sv and head_dim == dk == dq == dm == dv
            and n_kv_heads == n_v_heads):
        raise ValueError("q_proxy, k_proxy, q, k, and v must agree on batch, sequence, head dimension, "
                         "and KV head count")
    if s % BLOCK_SIZE != 0:
        raise ValueError(f"sequence length must be divisible by {BLOCK_SIZE}, got {s}")
    if n_proxy_heads % n_proxy_kv_heads != 0:
        raise ValueError("n_proxy_heads must be divisible by n_proxy_kv_heads")
    if n_heads % n_kv_heads != 0:
        raise ValueError("n_heads must be divisible by n_kv_heads")
    if n_heads % n_proxy_heads != 0:
        raise ValueError("n_heads must be divisible by n_proxy_heads")
    if head_dim != 128:
        raise NotImplementedError("Headdim must be 128")
    if n_proxy_heads < n_kv_heads or n_proxy_heads % n_kv_heads != 0:
        raise NotImplementedError("n_proxy_heads must be a multiple of n_kv_heads")
    dts = {t.dtype for t in (q_proxy, k_proxy, q, k, v)}
    if len(dts) != 1 or q.dtype not in (torch.bfloat16, torch.float16):
        raise TypeError(f"flash_msa_b200 supports bf16 or fp16 activations of one dtype, got {sorted(map(str, dts))}")
    num_blocks = s // BLOCK_SIZE
    if not sparse:
        return num_blocks, 0
    if int(top_k) % BLOCK_SIZE != 0:
        raise ValueError(f"top_k must be divisible by {BLOCK_SIZE}, got {top_k}")
    top_k_blocks = int(top_k) // BLOCK_SIZE
    if not 1 <= top_k_blocks <= num_blocks:
        raise ValueError(f"top_k selects {top_k_blocks} blocks, but sequence has {num_blocks} blocks")
    if top_k_blocks > MAX_TOP_K_BLOCKS:
        raise NotImplementedError(f"No more than {MAX_TOP_K_BLOCKS} blocks / topk={MAX_TOP_K_BLOCKS * BLOCK_SIZE} supported")
    return num_blocks, top_k_blocks


def _require_cuda(q, message="flash_msa_b200 requires CUDA tensors (there is no CPU path)"):
    if q.device.type != "cuda":
        raise RuntimeError(message)


# The reference returns a zero placeholder as kl_loss and users cannot watch the distillation loss
# (flash_msa/msa_forward_cutedsl.py:69).  With COMPUTE_KL_VALUE = True every backward that receives a
# gradient for kl_loss also computes the loss value inside the backward kernel (the teacher and the proxy
# probabilities are in registers there anyway); ``last_kl_value()`` returns it.
COMPUTE_KL_VALUE = False
_last_kl_value = None


def last_kl_value():
    """0-dim fp32 CUDA tensor: the KL loss of the most recent backward that ran with
    ``COMPUTE_KL_VALUE = True`` (mean over batch, proxy heads and rows of KL(teacher || proxy), the
    value of the reference's eager model, flash_msa/tests/testing_model.py:158-167).  None before the
    first such backward.  Reading it does not synchronise; ``.item()`` does."""
    return _last_kl_value


def _kl_buffer(grad_kl, device):
    if COMPUTE_KL_VALUE and grad_kl is not None:
        return torch.zeros(1, dtype=torch.float32, device=device)
    return None


def _publish_kl(buf):
    global _last_kl_value
    if buf is not None:
        _last_kl_value = buf.reshape(())


class _Status:
    """Status word of one call."""

    def __init__(self, kind, device):
        self.kind = kind
        if DEBUG_CHECK_STATUS:
            self.word = torch.zeros(1, dtype=torch.int32, device=device)
            self.ptr = self.word.data_ptr()
        else:
            self.word = None
            self.ptr = passes.status_board.pointer(kind, device)

    def check(self):
        if self.word is not None:
            ops.check_status(self.word, passes.StatusBoard.KINDS[self.kind])


def check_pending_status():
    """Waits for all calls issued so far and raises RuntimeError if one of them reported trouble."""
    passes.status_board.drain()


def _check_sinks(sinks, q):
    if sinks is None:
        return None
    if sinks.ndim != 1 or sinks.shape[0] != q.shape[1] or sinks.device != q.device:
        raise ValueError("sinks must hold one logit per main query head, on the inputs' device")
    return sinks


def _sink_logits(sinks):
    """fp32 contiguous logits as the kernels read them (a softmax bias, "attention sink": see fmsa_forward_args)."""
    return None if sinks is None else sinks.detach().to(torch.float32).contiguous()


def _forward(q_proxy, k_proxy, q, k, v, top_k, scale, sparse, doc_start, visible, sinks, with_proxy):
    """Checks the call, then runs its forward: (plan, fp32 sink logits or None, out, kl_loss placeholder, saved)."""
    _, top_k_blocks = _validate_inputs(q_proxy, k_proxy, q, k, v, top_k if sparse else 0, sparse)
    if sparse:
        _require_cuda(q)
    sinks = _check_sinks(sinks, q)
    if not sparse:
        _require_cuda(q, "warmup MSA forward requires CUDA tensors")
    inputs = (q_proxy, k_proxy, q, k, v)
    dev = q.device
    if q_proxy.device != dev or k_proxy.device != dev or k.device != dev or v.device != dev:   # (a host pointer would reach the kernels as it is)
        raise ValueError("q_proxy, k_proxy, q, k, and v must be on one CUDA device")
    plan = passes.plan(inputs, top_k_blocks, scale, not sparse)
    logits = _sink_logits(sinks)
    status = _Status(0 if sparse else 2, plan.device)
    out, kl_loss, saved = passes.forward(plan, inputs, doc_start, logits, status.ptr, with_proxy, *((visible,) if visible else ()))
    status.check()
    return plan, logits, out, kl_loss, saved


class _AttentionFunction(torch.autograd.Function):
    """Sparse or dense warmup attention behind autograd.  kl_loss is a placeholder whose gradient switches the KL branch of
    the backward on (reference: flash_msa/msa_forward_cutedsl.py:69)."""

    @staticmethod
    def forward(ctx, q_proxy, k_proxy, q, k, v, sinks, doc_start, visible, top_k, scale, sparse):
        # (everything that depends on the inputs is done in here: a trace records this call as one node, which comes back with
        # tensors of any size when the trace is run)
        plan, logits, out, kl_loss, saved = _forward(q_proxy, k_proxy, q, k, v, top_k, scale, sparse, doc_start, visible, sinks, True)
        ctx.save_for_backward(q_proxy, k_proxy, q, k, v, out, saved)
        # an output that does not feed the loss arrives as None in backward (not as zeros): no gradient for
        # kl_loss then really skips the proxy work, as the reference intends (flash_msa/flash_msa.py:104-106)
        ctx.set_materialize_grads(False)
        ctx.plan, ctx.doc_start, ctx.logits = plan, doc_start, logits
        ctx.sinks_dtype = None if sinks is None else sinks.dtype
        return out, kl_loss

    @staticmethod
    def backward(ctx, grad_out, grad_kl):
        q_proxy, k_proxy, q, k, v, out, saved = ctx.saved_tensors
        plan = ctx.plan
        if grad_out is None:
            grad_out = torch.zeros_like(out)
        status = _Status(3 if plan.dense else 1, plan.device)
        klv = _kl_buffer(grad_kl, plan.device)
        dqp, dkp, dq, dk, dv, dsinks = passes.backward(plan, (q_proxy, k_proxy, q, k, v), out, grad_out, saved, grad_kl, klv, ctx.doc_start,
                                                       ctx.logits, status.ptr)
        _publish_kl(klv)
        status.check()
        return dqp, dkp, dq, dk, dv, None if dsinks is None else dsinks.to(ctx.sinks_dtype), None, None, None, None, None


def _attend(q_proxy, k_proxy, q, k, v, top_k, scale, sparse, documents, sinks):
    doc_start, visible = documents
    q_proxy = _spread_proxy_heads(q_proxy, k_proxy, q, k)
    with_grad = torch.is_grad_enabled() and (q_proxy.requires_grad or k_proxy.requires_grad or q.requires_grad or k.requires_grad or
                                             v.requires_grad or (sinks is not None and sinks.requires_grad))
    if with_grad or forward_ad._current_level >= 0 or torch._C._is_tracing():
        return _AttentionFunction.apply(q_proxy, k_proxy, q, k, v, sinks, doc_start, visible, top_k, scale, sparse)
    # No backward will follow: the proxy log-sum-exp, which only the backward needs, is left out.  (Tangents would be lost
    # here, which the autograd function refuses, and a trace would hold nothing but the allocation of `out`.)
    return _forward(q_proxy, k_proxy, q, k, v, top_k, scale, sparse, doc_start, visible, sinks, False)[2:4]


def _spread_proxy_heads(q_proxy, k_proxy, q, k):
    """Fewer proxy heads than KV heads (Hkv % Hp == 0; the reference refuses this, flash_msa/flash_msa.py:44-62): the
    kernels walk one KV head at a time and want that head's proxy head(s) with it, so every proxy query head is
    repeated Hkv/Hp times (a differentiable copy of the small proxy tensor).  Each copy then steers the main heads of
    one KV head with the same scores, hence the same selection, and autograd sums the copies' gradients.  That sum is
    exact: the gradient of the KL term is linear in the teacher, the copies' teachers are the means over their own
    main heads, and the per-call factor 1/(B*Hp'*S) with Hp' = Hkv makes their sum the gradient for the mean over all
    main heads of the proxy head.  (Only the optional KL VALUE differs: it becomes the mean of the copies' KL terms,
    an upper bound of the KL against the pooled teacher.)"""
    if q_proxy.ndim == 4 and k_proxy.ndim == 4 and q.ndim == 4 and k.ndim == 4:
        hp, hpkv, hq, hkv = q_proxy.shape[1], k_proxy.shape[1], q.shape[1], k.shape[1]
        if 0 < hp < hkv and hkv % hp == 0 and hpkv > 0 and hp % hpkv == 0 and hq % hkv == 0:
            return q_proxy.repeat_interleave(hkv // hp, dim=1)
    return q_proxy   # (anything else is judged by the shape checks of the call)


_NO_DOCUMENTS = (None, 0)


def _documents(q, cu_seqlens):
    if q.ndim != 4:
        raise ValueError("all attention tensors must have shape (B, H, S, D)")
    _require_cuda(q)
    return ops.document_layout(cu_seqlens, q.shape[0], q.shape[2], q.device)


def sparse_attention(q_proxy, k_proxy, q, k, v, top_k: int, scale: float, sinks=None):
    """Block-sparse top-k GQA attention.  Returns ``(attn_out [B,S,Hq*D], kl_loss placeholder)``.
    ``sinks`` (optional, beyond the reference): one softmax-bias logit per main query head that joins the softmax
    denominator and contributes no value."""
    return _attend(q_proxy, k_proxy, q, k, v, int(top_k), float(scale), True, _NO_DOCUMENTS, sinks)


def sparse_attention_varlen(q_proxy, k_proxy, q, k, v, cu_seqlens, top_k: int, scale: float, sinks=None):
    """`sparse_attention` on packed sequences: the S positions of every batch element hold several documents laid end
    to end, `cu_seqlens` ([n+1], or [B,n+1] for a packing per batch element; starts at 0, ends at S: the FlashAttention
    varlen convention) gives their boundaries, and a query sees only the keys of its own document - in the block scores
    and the selection, in the attention and in every gradient.  Blocks stay 128 positions of the PACKED sequence, so S
    must still be a multiple of 128 (pad the last document).  The reference has no such path (its README lists
    variable-length batches as missing).  Boundaries in host memory (a list, a CPU tensor) are checked there
    and travel with a kernel launch; those in a CUDA tensor make the call wait for the device, for the same checks."""
    return _attend(q_proxy, k_proxy, q, k, v, int(top_k), float(scale), True, _documents(q, cu_seqlens), sinks)


def sparse_attention_warmup(q_proxy, k_proxy, q, k, v, top_k: int, scale: float, sinks=None):
    """Dense causal warmup attention with full-sequence proxy KL gradients (top_k is accepted and ignored, as in the
    reference)."""
    return _attend(q_proxy, k_proxy, q, k, v, int(top_k), float(scale), False, _NO_DOCUMENTS, sinks)


def sparse_attention_warmup_varlen(q_proxy, k_proxy, q, k, v, cu_seqlens, top_k: int, scale: float, sinks=None):
    """`sparse_attention_warmup` on packed sequences (see `sparse_attention_varlen`): dense causal attention and the
    full-sequence proxy KL inside every document.  The schedule still visits every causal block pair of the packed
    sequence; pairs that straddle documents are masked."""
    return _attend(q_proxy, k_proxy, q, k, v, int(top_k), float(scale), False, _documents(q, cu_seqlens), sinks)
