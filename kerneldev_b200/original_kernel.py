"""Host side of the attention operator: the call signature of the reference's
``original_kernel.flash_attention`` (original_kernel.py:2096-2168) in front of the hand-written
sm_100a kernels in libkd_attention.so.

``flash_attention`` is a drop-in for ``model.MultiHeadAttention`` (model.py:83-93): same
arguments, same return structure, O contiguous in the dtype of q (original_kernel.py:1801), LSE in base-2 units
(original_kernel.py:603-604), gradients for q, k and v only (the gradient of LSE is ignored,
as at original_kernel.py:1965-1992).

Differences from the reference, all deliberate:
  * the mask is the rule of original_kernel.py:480-517 for the forward AND the backward; the
    reference's backward loop bounds ignore the bidirectional sections when ``causal=True`` and
    metadata is given (original_kernel.py:1202-1204, :1368-1371);
  * a query row that sees no key gets O = 0, LSE = -inf and no gradient (the reference's default
    path produces NaN there, original_kernel.py:554-561);
  * CUDA sm_100 only, fp16 / bf16 (fp32 tensors as fp16 operands), head_dim a multiple of 16 up to 128 (the reference also
    takes 256). There is no Triton, no autotuning and no CPU path: unsupported inputs raise, as do forward-mode AD and
    tracing.
``autotune``, ``prescale_qk`` and ``precision`` are accepted and ignored.
"""
from __future__ import annotations

import torch

from . import _capi, _host
from .plan import AttentionPlan, get_plan

_ext = _host.load()  # fails at import time, loudly, when the CUDA library or the host extension has not been built

__all__ = ["flash_attention", "generate_hadamard_signs", "hadamard_transform"]

_HADAMARD_DIMS = (16, 32, 64, 128)
_DTYPES = {torch.float16: _capi.KD_F16, torch.bfloat16: _capi.KD_BF16}


def _kd_tensor(t: torch.Tensor) -> _capi.KdTensor:
    return _capi.KdTensor(t.data_ptr(), t.stride(0), t.stride(1), t.stride(2))


def _params(q, k, v, o, lse, plan, sm_scale):
    B, H, T, D = q.shape
    p = _capi.KdAttnParams()
    p.B, p.H, p.T, p.D = B, H, T, D
    p.dtype = _DTYPES[q.dtype]
    p.sm_scale = sm_scale
    p.q, p.k, p.v, p.o = _kd_tensor(q), _kd_tensor(k), _kd_tensor(v), _kd_tensor(o)
    p.lse = lse.data_ptr()
    p.plan = plan.ptr
    return p


def _forward(q, k, v, plan: AttentionPlan, sm_scale: float, like_input: bool = False):
    """One kd_attn_fwd call: returns (O, LSE) for inputs flash_attention would accept. ``like_input``: O in the
    memory layout of q instead of contiguous."""
    return _ext.forward(q, k, v, plan._core, sm_scale, like_input)


def _backward(q, k, v, o, lse, d_o, plan: AttentionPlan, sm_scale: float, phases: int = 0, bufs=None,
              like_input: bool = False, deterministic: bool = False):
    """One kd_attn_bwd call: returns (dQ, dK, dV). ``phases`` selects a part of the backward (see
    kd_attn_params.bwd_phases); ``bufs`` = (dq, dk, dv, delta[, dq_acc]) reuses buffers.
    ``deterministic=False`` selects the fused backward: one pass over the tiles instead of two, dQ accumulated
    with fp32 additions in a scratch (kd_workspace_bytes_fused)."""
    return _ext.backward(q, k, v, o, lse, d_o, plan._core, sm_scale, phases, list(bufs or ()), like_input, deterministic)


def _hadamard_call(x: torch.Tensor, signs, inverse: bool) -> torch.Tensor:
    return _ext.hadamard(x, signs, inverse)


class _HadamardFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, signs):
        ctx.signs = signs
        return _hadamard_call(x, signs, inverse=False)

    @staticmethod
    def backward(ctx, dy):
        # y = x diag(s) W / sqrt(D) with W symmetric, so dx = dy W / sqrt(D) diag(s)
        return _hadamard_call(dy, ctx.signs, inverse=True), None


def generate_hadamard_signs(n_heads: int, head_dim: int, seed: int = 0, device="cuda") -> torch.Tensor:
    """(n_heads, head_dim) float32 tensor of +-1 drawn from a seeded CPU generator.

    The reference only names this utility (README.md:68-77); the recipe here is this package's own:
    ``torch.randint(0, 2, (n_heads, head_dim), generator=torch.Generator().manual_seed(seed)) * 2 - 1``.
    """
    g = torch.Generator(device="cpu").manual_seed(seed)
    s = torch.randint(0, 2, (n_heads, head_dim), generator=g, dtype=torch.int64) * 2 - 1
    return s.to(torch.float32).to(device)


def _check_signs(signs: torch.Tensor, n_heads: int, head_dim: int, device) -> torch.Tensor:
    if signs.shape != (n_heads, head_dim):
        raise ValueError("signs must have shape (heads, head_dim)")
    signs = signs.to(device=device, dtype=torch.float32).contiguous()
    return signs if signs.data_ptr() % 16 == 0 else signs.clone()   # the kernels read four at a time


def hadamard_transform(x: torch.Tensor, signs: torch.Tensor | None = None) -> torch.Tensor:
    """``WHT(x * signs[h]) / sqrt(D)`` over the last dimension of a (B, H, T, D) tensor, with the
    Walsh-Hadamard matrix in natural (Sylvester) order; differentiable."""
    if x.dim() != 4 or x.shape[-1] not in _HADAMARD_DIMS or x.dtype not in _DTYPES or not x.is_cuda:
        raise ValueError("hadamard_transform expects a CUDA (B, H, T, D) fp16/bf16 tensor with D in {16, 32, 64, 128}")
    if signs is not None:
        signs = _check_signs(signs, x.shape[1], x.shape[3], x.device)
    return _HadamardFn.apply(x, signs)


def flash_attention(
    q: torch.Tensor,
    k: torch.Tensor,
    v: torch.Tensor,
    lens: torch.Tensor | None = None,
    sm_scale: float | None = None,
    causal: bool = True,
    autotune=False,
    return_lse=False,
    prescale_qk=False,
    precision="tf32",
    attention_mask: torch.Tensor | None = None,
    in_span: torch.Tensor | None = None,
    span_id: torch.Tensor | None = None,
    is_prefix: torch.Tensor | None = None,
    return_attention_mask: bool = False,
    hadamard_signs: torch.Tensor | None = None,
    out_layout: str = "contiguous",
    deterministic: bool = False,
):
    """Self-attention with the 4-section hierarchical mask; arguments and return value as the
    reference's ``flash_attention`` (original_kernel.py:2096-2168).

    q, k, v: (batch, heads, time, head_dim), any strides. lens: int32 (batch,) or None.
    in_span / is_prefix: bool (batch, time); span_id: int64 (batch, time) (1-based span ids, -1 at
    [MASKQ]). When any of attention_mask / in_span / span_id / is_prefix is given the mask is the
    rule of original_kernel.py:480-517 and ``causal`` is not part of it; otherwise the mask is
    ``i >= j`` (causal) or all-ones. ``attention_mask`` itself is never read (as in the reference).

    hadamard_signs (extension, default None): (heads, head_dim) +-1; Q and K are replaced by
    ``hadamard_transform(., signs)`` before the attention, which leaves Q K^T unchanged in exact
    arithmetic and spreads outliers over the head dimension.
    out_layout (extension): "contiguous" (default, as original_kernel.py:1801 and :1920-1922) or
    "input": O and the gradients take the memory layout of q, k, v. For the model's (B,H,T,D) views
    of (B,T,H,D) memory (model.py:76-78) the ``transpose(1, 2).contiguous()`` after the call
    (model.py:95) and its counterpart in the backward then copy nothing. The drop-in module uses it.
    deterministic (extension, default False): True forces the two-kernel backward, whose results are
    bit-identical from run to run and which needs no scratch beyond 4 bytes a row; the default, at every head dim, is the
    fused backward, which forms S and dP once per tile and adds dQ partials in fp32 in no fixed order (dQ then varies in its
    last bits between runs) to a scratch of batch * heads * time rows of 64 floats (head_dim <= 64) or 128 (above).

    float32 q, k, v (the reference's default ``precision="tf32"`` path, original_kernel.py:2106): the tensors
    are rounded to float16 operands -- the 10-bit mantissa tf32 keeps -- the products accumulate in fp32 as
    everywhere, and O and the gradients come back as float32. Values must lie inside float16's range
    (|x| < 65504; tf32 keeps fp32's exponent). ``precision="ieee"`` with float32 tensors is not supported.

    Returns O, or (O, LSE) with return_lse, or (that, mask[B,H,T,T] bool) with return_attention_mask.
    """
    if precision == "ieee" and q.dtype is torch.float32 and k.dtype is torch.float32 and v.dtype is torch.float32:
        raise ValueError("float32 inputs with precision='ieee' are not supported: the tensor cores take 16-bit operands here "
                         "(precision='tf32' rounds the operands to tf32's 10-bit mantissa)")
    if out_layout not in ("contiguous", "input"):
        raise ValueError("out_layout must be 'contiguous' or 'input'")
    rules = attention_mask is not None or in_span is not None or span_id is not None or is_prefix is not None
    if hadamard_signs is not None and q.dim() == 4:
        if q.shape[-1] not in _HADAMARD_DIMS:
            raise ValueError("hadamard_signs needs a head_dim in {16, 32, 64, 128}")
        hadamard_signs = _check_signs(hadamard_signs, q.shape[1], q.shape[3], q.device)
    o, lse = _ext.attention(q, k, v, lens, sm_scale, bool(causal), in_span, span_id, is_prefix, rules, hadamard_signs,
                            out_layout == "input", bool(deterministic), bool(return_lse))

    if return_attention_mask:
        B, H, T, _ = q.shape
        plan = get_plan(B, T, q.device, in_span, span_id, is_prefix, lens, causal, rules)
        mask = plan.dense_mask().unsqueeze(1).expand(B, H, T, T)
        if return_lse:
            return (o, lse), mask
        return o, mask
    if return_lse:
        return o, lse
    return o
