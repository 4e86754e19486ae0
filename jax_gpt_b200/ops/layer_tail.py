"""Ends of a layer in one launch (csrc/layer_tail.cu): inference only, bf16 on CUDA."""
from __future__ import annotations

from typing import Optional

import torch

from .. import _ext

MAX_WIDTH = 8192


def tail_ok(*tensors) -> bool:
    """Whether rows of these (bf16 activations and weights) can go through ``layer_tail``: plain CUDA tensors, widths in 16-byte
    pieces, and nothing that wants a gradient."""
    return all(torch.is_tensor(t) and t.is_cuda and t.dtype == torch.bfloat16 and t.is_contiguous() and t.data_ptr() % 16 == 0 for t in tensors) \
        and tensors[0].shape[-1] % 8 == 0 and tensors[0].shape[-1] <= MAX_WIDTH \
        and not (torch.is_grad_enabled() and any(t.requires_grad for t in tensors))


def layer_tail(x=None, routed=None, shared=None, h=None, gate_w=None, norm_w=None, eps: float = 1e-6, one_plus: bool = True):
    """``x + routed + shared * sigmoid(h . gate_w)`` of rows (M, D), rounded once, and with ``norm_w`` also its RMS norm: returns the
    sum, or (sum, norm). ``routed`` is fp32, the others bf16; what is None is left out, without ``gate_w`` shared counts as it is."""
    like = x if x is not None else shared
    out = torch.empty_like(like)
    normed = torch.empty_like(like) if norm_w is not None else None
    _ext.ops().layer_tail(x, routed, shared, h, None if gate_w is None else gate_w.reshape(-1), norm_w, eps, one_plus, out, normed)
    return out if normed is None else (out, normed)


def layer_tail_ref(x=None, routed=None, shared=None, h=None, gate_w=None, norm_w=None, eps: float = 1e-6, one_plus: bool = True):
    like = x if x is not None else shared
    v = torch.zeros(like.shape, device=like.device)
    if x is not None:
        v = v + x.float()
    if routed is not None:
        v = v + routed
    if shared is not None:
        v = v + shared.float() * (1.0 if gate_w is None else torch.sigmoid(h.float() @ gate_w.float().reshape(-1, 1)))
    out = v.to(like.dtype)
    if norm_w is None:
        return out
    f = out.float()
    return out, (f * torch.rsqrt(f.square().mean(-1, keepdim=True) + eps) * (norm_w.float() + (1.0 if one_plus else 0.0))).to(like.dtype)


def silu_mul(g: torch.Tensor, u: torch.Tensor) -> torch.Tensor:
    """``silu(g) * u``; without gradients in bf16 on CUDA one launch with one rounding (g and u may be column slices)."""
    n = g.shape[-1]
    piece = lambda t: (t.is_cuda and t.dtype == torch.bfloat16 and t.dim() == 2 and t.stride(1) == 1 and t.stride(0) % 8 == 0
                       and t.data_ptr() % 16 == 0)
    if not (g.shape == u.shape and n % 8 == 0 and piece(g) and piece(u)) or (torch.is_grad_enabled() and (g.requires_grad or u.requires_grad)):
        return torch.nn.functional.silu(g) * u
    out = torch.empty(g.shape, device=g.device, dtype=g.dtype)
    _ext.ops().silu_mul(g, u, out)
    return out


def gate_heads(o: torch.Tensor, qg: torch.Tensor) -> torch.Tensor:
    """``o * sigmoid(gate)`` with qg (..., 2 d) = [query | gate] per head of o (..., d); in place where nothing wants a gradient."""
    d = o.shape[-1]
    if tail_ok(o) and qg.dtype == o.dtype and not (torch.is_grad_enabled() and qg.requires_grad):
        _ext.ops().sigmoid_gate(o.view(-1, d), qg.reshape(-1, 2 * d)[:, d:])
        return o
    return o * torch.sigmoid(qg[..., d:].float()).to(o.dtype)


def argmax_rows(x: torch.Tensor, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Place of the largest of every row of x (rows, N), the first of equal ones; int64."""
    if not (x.is_cuda and x.dtype == torch.bfloat16 and x.dim() == 2 and x.stride(1) == 1):
        best = x.argmax(-1)
        return best if out is None else out.copy_(best)
    if out is None:
        out = torch.empty(x.shape[0], device=x.device, dtype=torch.long)
    _ext.ops().argmax_rows(x, out)
    return out
