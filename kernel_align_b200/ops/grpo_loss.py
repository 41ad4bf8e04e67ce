"""GRPO objective: group-normalised advantages and the clipped-ratio policy loss.

CUDA: ``csrc/sm100/grpo_loss.cu`` (fixed-order reductions, bitwise reproducible loss) behind the C++ autograd node of
``csrc/torch/grpo_autograd.cpp``, or behind the Python one below where that module is not there (a package built without torch),
which costs the host 31 us more for advantages, loss and gradient (108 against 77); CPU: ``csrc/cpu/grpo_loss_cpu.cpp``.
``grpo_loss`` is differentiable with respect to ``logp_new``. The reference lists the GRPO loss in its README but ships no implementation.
"""
from __future__ import annotations

from ctypes import c_float, c_int, c_void_p
from typing import Optional

import torch

from .. import _native
from ..utils.profiler import profiled


def group_advantages(rewards: torch.Tensor, group_size: int, eps: float = 1e-4) -> torch.Tensor:
    """``(r - mean_group) / (std_group + eps)`` over consecutive groups of ``group_size``
    rewards (unbiased standard deviation)."""
    if rewards.numel() % group_size:
        raise ValueError("the number of rewards must be a multiple of the group size")
    cuda = rewards.device.type == "cuda"
    if cuda and (node := _native.torch_ops()) is not None:
        return node.group_advantages(rewards, group_size, eps)
    r = rewards.reshape(-1).float().contiguous()
    adv = torch.empty_like(r)
    n_groups = r.numel() // group_size
    if cuda:
        rc = _native.cuda().ka_grpo_advantages(r.data_ptr(), adv.data_ptr(), n_groups, group_size, eps,
                                               _native.stream_ptr(r.device))
    else:
        fn = _native.cpu().ka_cpu_grpo_advantages
        fn.restype = c_int
        fn.argtypes = [c_void_p, c_void_p, c_int, c_int, c_float]
        rc = fn(r.data_ptr(), adv.data_ptr(), n_groups, group_size, eps)
    if rc != 0:
        raise RuntimeError(f"grpo advantages failed ({rc})")
    return adv.reshape(rewards.shape)


class _GrpoLossFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, logp_new, logp_old, logp_ref, adv, mask, eps_low, eps_high, beta, seq_mean, with_stats):
        ctx.set_materialize_grads(False)
        n_seq, seq_len = logp_new.shape
        ln = logp_new.float().contiguous()
        lo = logp_old.float().contiguous()
        lr = logp_ref.float().contiguous() if logp_ref is not None else None
        a = adv.float().contiguous()
        ctx.shape = (n_seq, seq_len)
        ctx.cuda = ln.device.type == "cuda"
        if ctx.cuda:
            # bytes and floats are read as they are, anything else is converted first
            if mask is not None and mask.dtype not in (torch.bool, torch.uint8, torch.float32):
                mask = mask.to(torch.uint8)
            m = mask.contiguous() if mask is not None else None
            if any(t is not None and t.device != ln.device for t in (lo, lr, a, m)):
                raise RuntimeError("the GRPO operators take tensors that are all on the CPU or all on a CUDA device")
            raw = torch.empty_like(ln)
            ws = torch.empty(4 * n_seq + 3, dtype=torch.float32, device=ln.device)   # per sequence, then the statistics
            loss = torch.empty((), dtype=torch.float32, device=ln.device)
            out = torch.empty(3, dtype=torch.float32, device=ln.device) if with_stats else None
            rc = _native.cuda().ka_grpo_loss_fwd(
                ln.data_ptr(), lo.data_ptr(), lr.data_ptr() if lr is not None else None, a.data_ptr(),
                m.data_ptr() if m is not None else None, int(m is not None and m.dtype == torch.float32), n_seq,
                seq_len, eps_low, eps_high, beta, int(seq_mean), raw.data_ptr(), ws.data_ptr(), loss.data_ptr(),
                out.data_ptr() if with_stats else ws.data_ptr() + 16 * n_seq, _native.stream_ptr(ln.device))
            if rc != 0:
                raise RuntimeError(f"ka_grpo_loss_fwd failed ({rc})")
            ctx.save_for_backward(raw, ws)
            if not with_stats:
                return loss
            ctx.mark_non_differentiable(out)
            return loss, out
        m = mask.to(torch.uint8).contiguous() if mask is not None else None
        grad = torch.empty_like(ln)
        out = torch.empty(3, dtype=torch.float32, device=ln.device)
        fn = _native.cpu().ka_cpu_grpo_loss
        fn.restype = c_int
        fn.argtypes = [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_float, c_float, c_float,
                       c_int, c_void_p, c_void_p]
        rc = fn(ln.data_ptr(), lo.data_ptr(), lr.data_ptr() if lr is not None else None, a.data_ptr(),
                m.data_ptr() if m is not None else None, n_seq, seq_len, eps_low, eps_high, beta, int(seq_mean),
                grad.data_ptr(), out.data_ptr())
        if rc != 0:
            raise RuntimeError(f"ka_cpu_grpo_loss failed ({rc})")
        ctx.save_for_backward(grad)
        if not with_stats:
            return out[0].clone()
        ctx.mark_non_differentiable(out)
        return out[0].clone(), out

    @staticmethod
    def backward(ctx, g_loss, _g_stats=None):
        if g_loss is None:
            return (None,) * 10
        n_seq, seq_len = ctx.shape
        if ctx.cuda:
            raw, ws = ctx.saved_tensors
            grad = torch.empty_like(raw)
            up = g_loss.float().contiguous()
            rc = _native.cuda().ka_grpo_loss_bwd(raw.data_ptr(), ws.data_ptr() + 12 * n_seq, up.data_ptr(),
                                                 grad.data_ptr(), n_seq, seq_len, _native.stream_ptr(raw.device))
            if rc != 0:
                raise RuntimeError(f"ka_grpo_loss_bwd failed ({rc})")
        else:
            (g,) = ctx.saved_tensors
            grad = g * g_loss
        return (grad,) + (None,) * 9


@profiled("grpo_loss")
def grpo_loss(logp_new: torch.Tensor, logp_old: torch.Tensor, advantages: torch.Tensor, *,
              mask: Optional[torch.Tensor] = None, logp_ref: Optional[torch.Tensor] = None, eps_low: float = 0.2,
              eps_high: Optional[float] = None, beta: float = 0.0, reduction: str = "token_mean",
              return_stats: bool = False):
    """Clipped-ratio GRPO loss. ``logp_*`` ``[G, L]`` fp32, ``advantages`` ``[G]``, ``mask`` ``[G, L]``.

    ``reduction``: ``"token_mean"`` (mean over all valid tokens) or ``"seq_mean"`` (mean over
    sequences of their token means). With ``return_stats`` also returns a tensor
    ``[loss, clip_fraction, valid_tokens]``.
    """
    if reduction not in ("token_mean", "seq_mean"):
        raise ValueError("reduction must be 'token_mean' or 'seq_mean'")
    hi = eps_low if eps_high is None else eps_high
    args = (logp_new, logp_old, logp_ref, advantages, mask, float(eps_low), float(hi), float(beta),
            reduction == "seq_mean", bool(return_stats))
    if logp_new.device.type != "cuda" or (node := _native.torch_ops()) is None:
        return _GrpoLossFn.apply(*args)
    if logp_new.dim() != 2:
        raise ValueError("logp_new must be [sequences, tokens]")
    out = node.grpo_loss(*args)
    return tuple(out) if return_stats else out[0]
