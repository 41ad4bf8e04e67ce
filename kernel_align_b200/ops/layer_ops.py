"""RMSNorm (with fused residual add), rotary embedding and SwiGLU.

CUDA: ``csrc/sm100/elementwise.cu`` (bf16 in/out, fp32 math, fixed-order reductions, one pass).
CPU: ``csrc/cpu/layer_ops_cpu.cpp`` with the same rounding points. The reference only names
these ops (README feature list, ``ActivationFunction.SILU`` in
rl_engine/platforms/constants.py:75-80).
"""
from __future__ import annotations

from ctypes import c_float, c_int, c_longlong, c_void_p
from typing import Optional

import torch

from .. import _native
from ..utils.profiler import profiled


def _sms(t: torch.Tensor) -> int:
    return _native.sm_count(t.device)


def _stream(t: torch.Tensor) -> int:
    return _native.stream_ptr(t.device)


def _packed(t: torch.Tensor) -> torch.Tensor:
    """``t`` contiguous and 16-byte aligned. Gradients come from anywhere: a piece of a packed buffer
    is contiguous, but may start at any element, and the kernels read 16 bytes at a time."""
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


def _check(rc: int, name: str) -> None:
    if rc != 0:
        raise RuntimeError(f"{name} failed ({rc})")


@profiled("rmsnorm")
def rmsnorm(x: torch.Tensor, weight: torch.Tensor, eps: float = 1e-5, residual: Optional[torch.Tensor] = None):
    """``y = rmsnorm(x + residual) * weight``. With ``residual`` returns ``(y, x + residual)``."""
    d = x.shape[-1]
    x2 = x.reshape(-1, d)
    rows = x2.shape[0]
    if x.device.type != "cuda":
        lib = _native.cpu()
        xf = x2.float().contiguous()
        rf = residual.reshape(-1, d).float().contiguous() if residual is not None else None
        wf = weight.float().contiguous()
        y = torch.empty_like(xf)
        ro = torch.empty_like(xf) if residual is not None else None
        fn = lib.ka_cpu_rmsnorm
        fn.restype = c_int
        fn.argtypes = [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_float]
        _check(fn(xf.data_ptr(), rf.data_ptr() if rf is not None else None, wf.data_ptr(), y.data_ptr(),
                  ro.data_ptr() if ro is not None else None, rows, d, float(eps)), "ka_cpu_rmsnorm")
        y = y.to(x.dtype).reshape(x.shape)
        return (y, ro.to(x.dtype).reshape(x.shape)) if residual is not None else y
    if x.dtype != torch.bfloat16:
        raise TypeError("the sm_100a rmsnorm takes bf16")
    x2 = x2.contiguous()
    r2 = residual.reshape(-1, d).contiguous() if residual is not None else None
    y = torch.empty_like(x2)
    ro = torch.empty_like(x2) if residual is not None else None
    fn = _native.cuda().ka_rmsnorm
    _check(fn(x2.data_ptr(), r2.data_ptr() if r2 is not None else None, weight.contiguous().data_ptr(), y.data_ptr(),
              ro.data_ptr() if ro is not None else None, rows, d, float(eps), _sms(x), _stream(x)), "ka_rmsnorm")
    y = y.reshape(x.shape)
    return (y, ro.reshape(x.shape)) if residual is not None else y


def rope_tables(max_pos: int, head_dim: int, theta: float = 500000.0, device="cpu"):
    """``cos``/``sin`` tables ``[max_pos, head_dim/2]`` fp32, computed in float64 on the host so
    that every device sees the same values."""
    inv = 1.0 / (theta ** (torch.arange(0, head_dim, 2, dtype=torch.float64) / head_dim))
    ang = torch.arange(max_pos, dtype=torch.float64)[:, None] * inv[None, :]
    return ang.cos().float().to(device), ang.sin().float().to(device)


@profiled("rope")
def rope_(x: torch.Tensor, positions: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor) -> torch.Tensor:
    """Rotate ``x`` ``[tokens, heads, head_dim]`` in place ("rotate half" convention)."""
    tokens, heads, hd = x.shape
    pos = positions.reshape(-1).to(torch.int64).contiguous()
    if x.device.type != "cuda":
        lib = _native.cpu()
        xf = x.float().contiguous()
        fn = lib.ka_cpu_rope
        fn.restype = c_int
        fn.argtypes = [c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int]
        _check(fn(xf.data_ptr(), pos.data_ptr(), cos.contiguous().data_ptr(), sin.contiguous().data_ptr(), tokens,
                  heads, hd), "ka_cpu_rope")
        x.copy_(xf.to(x.dtype))
        return x
    if x.dtype != torch.bfloat16 or x.stride(2) != 1 or x.stride(1) != hd:
        raise ValueError("rope_ takes bf16 [tokens, heads, head_dim] with contiguous heads")
    fn = _native.cuda().ka_rope
    _check(fn(x.data_ptr(), x.stride(0), pos.data_ptr(), cos.data_ptr(), sin.data_ptr(), tokens, heads, hd, _sms(x),
              _stream(x)), "ka_rope")
    return x


@profiled("swiglu")
def swiglu(gate_up: torch.Tensor, up: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``silu(gate) * up``. Either one ``[..., 2F]`` tensor holding ``[gate | up]`` or two ``[..., F]``."""
    if up is None:
        f = gate_up.shape[-1] // 2
        g2 = gate_up.reshape(-1, 2 * f)
        gate_v, up_v, stride = g2[:, :f], g2[:, f:], 2 * f
        lead = gate_up.shape[:-1]
    else:
        f = gate_up.shape[-1]
        gate_v, up_v, stride = gate_up.reshape(-1, f).contiguous(), up.reshape(-1, f).contiguous(), f
        lead = gate_up.shape[:-1]
    rows = gate_v.shape[0]
    if gate_up.device.type != "cuda":
        lib = _native.cpu()
        gf, uf = gate_v.float().contiguous(), up_v.float().contiguous()
        out = torch.empty_like(gf)
        fn = lib.ka_cpu_swiglu
        fn.restype = c_int
        fn.argtypes = [c_void_p, c_void_p, c_void_p, c_longlong]
        _check(fn(gf.data_ptr(), uf.data_ptr(), out.data_ptr(), gf.numel()), "ka_cpu_swiglu")
        return out.to(gate_up.dtype).reshape(*lead, f)
    if gate_up.dtype != torch.bfloat16:
        raise TypeError("the sm_100a swiglu takes bf16")
    if up is None and not gate_up.is_contiguous():
        return swiglu(gate_up.contiguous())
    out = torch.empty(rows, f, dtype=torch.bfloat16, device=gate_up.device)
    fn = _native.cuda().ka_swiglu
    _check(fn(gate_v.data_ptr(), up_v.data_ptr(), stride, out.data_ptr(), rows, f, _sms(out), _stream(out)),
           "ka_swiglu")
    return out.reshape(*lead, f)


# --------------------------------------------------------------------------------------------
# Differentiable wrappers: on CUDA forward and backward both run the hand-written kernels; on
# CPU the forward is the C++ library and the backward the same formulas in PyTorch fp32.
# --------------------------------------------------------------------------------------------
def _rmsnorm_backward(x, weight, eps, dy, d_res):
    """``(dx, dw)`` of RMSNorm; ``d_res`` (or None) is added to the rounded ``dx``."""
    d = x.shape[-1]
    x2 = _packed(x.reshape(-1, d))
    dy2 = _packed(dy.reshape(-1, d))
    rows = x2.shape[0]
    if x.device.type != "cuda":
        xf, gf, wf = x2.float(), dy2.float(), weight.float()
        r = torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + eps)
        gw = gf * wf
        dx = r * gw - xf * (r.pow(3) * (gw * xf).mean(-1, keepdim=True))
        dw = (gf * xf * r).sum(0)
        dx = dx.to(x.dtype).reshape(x.shape)
        return (dx if d_res is None else dx + d_res), dw.to(weight.dtype)
    return _rmsnorm_backward_launch(x2, _packed(weight), eps, dy2,
                                    _packed(d_res.reshape(-1, d)) if d_res is not None else None, x.shape)


def _rmsnorm_backward_launch(x2, weight, eps, dy2, res2, shape):
    rows, d = x2.shape
    dx = torch.empty_like(x2)
    dw = torch.empty_like(weight)
    chunk = int(_native.cuda().ka_rmsnorm_bwd_chunk())
    part = torch.empty((rows + chunk - 1) // chunk, d, dtype=torch.float32, device=x2.device)
    fn = _native.cuda().ka_rmsnorm_bwd
    _check(fn(x2.data_ptr(), weight.data_ptr(), dy2.data_ptr(), res2.data_ptr() if res2 is not None else None,
              dx.data_ptr(), dw.data_ptr(), part.data_ptr(), rows, d, float(eps), _stream(x2)), "ka_rmsnorm_bwd")
    return dx.reshape(shape), dw


class _RMSNormFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight, eps):
        ctx.save_for_backward(x, weight)
        ctx.eps = eps
        return rmsnorm(x, weight, eps)

    @staticmethod
    def backward(ctx, dy):
        x, weight = ctx.saved_tensors
        return (*_rmsnorm_backward(x, weight, ctx.eps, dy, None), None)


def rmsnorm_fn(x: torch.Tensor, weight: torch.Tensor, eps: float = 1e-5) -> torch.Tensor:
    """Differentiable RMSNorm (no fused residual; add the residual with ``+`` before it)."""
    if not (x.requires_grad or weight.requires_grad) or not torch.is_grad_enabled():
        return rmsnorm(x, weight, eps)
    return _RMSNormFn.apply(x, weight, eps)


class _RMSNormForkFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight, eps):
        ctx.set_materialize_grads(False)
        ctx.save_for_backward(x, weight)
        ctx.eps = eps
        return rmsnorm(x, weight, eps), x.view_as(x)

    @staticmethod
    def backward(ctx, dy, d_res):
        x, weight = ctx.saved_tensors
        if dy is None:
            return d_res, None, None
        return (*_rmsnorm_backward(x, weight, ctx.eps, dy, d_res), None)


def rmsnorm_fork_fn(x: torch.Tensor, weight: torch.Tensor, eps: float = 1e-5):
    """``(rmsnorm(x) * weight, x)`` for a residual stream that goes both through the norm and past
    it. Backward adds the two gradients of ``x`` inside the norm's kernel."""
    if not (x.requires_grad or weight.requires_grad) or not torch.is_grad_enabled():
        return rmsnorm(x, weight, eps), x
    return _RMSNormForkFn.apply(x, weight, eps)


class _RopeFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, positions, cos, sin):
        ctx.save_for_backward(positions, cos, sin)
        return rope_(x.clone(memory_format=torch.contiguous_format), positions, cos, sin)

    @staticmethod
    def backward(ctx, dy):
        positions, cos, sin = ctx.saved_tensors
        # the transpose of a rotation is the rotation by the opposite angle
        return rope_(dy.contiguous().clone(), positions, cos, -sin), None, None, None


def rope_fn(x: torch.Tensor, positions: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor) -> torch.Tensor:
    """Out-of-place, differentiable rotary embedding of ``x`` ``[tokens, heads, head_dim]``."""
    return _RopeFn.apply(x, positions, cos, sin)


@profiled("rope")
def _qkv_rope_launch(qkv, positions, cos, sin, q, k, v, tokens, backward):
    fn = _native.cuda().ka_qkv_rope
    _check(fn(qkv.data_ptr(), qkv.stride(0), qkv.shape[1], positions.data_ptr(), cos.data_ptr(), sin.data_ptr(),
              q.data_ptr(), k.data_ptr(), v.data_ptr(), qkv.shape[0], tokens, q.shape[1], k.shape[1], int(backward),
              _stream(qkv)), "ka_qkv_rope")


class _QkvRopeFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, qkv, positions, cos, sin, hq, hkv, tokens):
        pos = positions.reshape(-1).to(torch.int64).contiguous()
        ctx.save_for_backward(pos, cos, sin)
        ctx.shape = qkv.shape
        q, k, v = (torch.empty(tokens, h, 128, dtype=qkv.dtype, device=qkv.device) for h in (hq, hkv, hkv))
        _qkv_rope_launch(qkv, pos, cos, sin, q, k, v, tokens, False)
        return q, k, v

    @staticmethod
    def backward(ctx, dq, dk, dv):
        pos, cos, sin = ctx.saved_tensors
        dqkv = torch.empty(ctx.shape, dtype=dq.dtype, device=dq.device)
        _qkv_rope_launch(dqkv, pos, _packed(cos), _packed(sin), _packed(dq), _packed(dk), _packed(dv), dq.shape[0], True)
        return dqkv, None, None, None, None, None, None


def _qkv_rope_takes(qkv, positions, cos, sin, tokens, head_dim) -> bool:
    """Whether the fused kernel takes these tensors: it reads everything 16 bytes at a time."""
    def table(t):
        return (t.device == qkv.device and t.dtype == torch.float32 and t.dim() == 2 and t.shape[1] == head_dim // 2
                and t.is_contiguous() and t.data_ptr() % 16 == 0)

    return (qkv.device.type == "cuda" and qkv.dtype == torch.bfloat16 and head_dim == 128 and tokens > 0
            and qkv.stride(1) == 1 and qkv.stride(0) % 8 == 0 and qkv.stride(0) >= qkv.shape[1]
            and qkv.data_ptr() % 16 == 0 and positions.device == qkv.device and table(cos) and table(sin))


def qkv_rope_fn(qkv: torch.Tensor, positions: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor, hq: int, hkv: int,
                head_dim: int, tokens: Optional[int] = None):
    """Cut a fused projection ``[rows, (hq + 2 hkv) * head_dim]`` into ``q``, ``k`` (rotated at the
    first ``tokens`` of ``positions``; all of them by default) and ``v``, each
    ``[tokens, heads, head_dim]``; rows past ``tokens`` are padding. Differentiable; the bits of
    slicing and :func:`rope_fn`, in one launch per direction."""
    positions = positions.reshape(-1)
    tokens = positions.numel() if tokens is None else int(tokens)
    if positions.numel() < tokens:
        raise ValueError(f"{positions.numel()} positions for {tokens} tokens")
    if qkv.dim() != 2 or qkv.shape[1] != (hq + 2 * hkv) * head_dim or qkv.shape[0] < tokens:
        raise ValueError(f"a projection of {tuple(qkv.shape)} for {tokens} tokens of {hq} + 2 * {hkv} heads of {head_dim}")
    positions = positions[:tokens]
    if _qkv_rope_takes(qkv, positions, cos, sin, tokens, head_dim):
        return _QkvRopeFn.apply(qkv, positions, cos, sin, hq, hkv, tokens)
    q = qkv[:tokens, : hq * head_dim].reshape(tokens, hq, head_dim)
    k = qkv[:tokens, hq * head_dim:(hq + hkv) * head_dim].reshape(tokens, hkv, head_dim)
    v = qkv[:tokens, (hq + hkv) * head_dim:].reshape(tokens, hkv, head_dim)
    return rope_fn(q, positions, cos, sin), rope_fn(k, positions, cos, sin), v


class _SwigluFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, gate_up):
        ctx.save_for_backward(gate_up)
        return swiglu(gate_up)

    @staticmethod
    def backward(ctx, d_out):
        (gate_up,) = ctx.saved_tensors
        f = gate_up.shape[-1] // 2
        gu = gate_up.reshape(-1, 2 * f)
        d2 = d_out.reshape(-1, f).contiguous()
        rows = gu.shape[0]
        if gate_up.device.type != "cuda":
            g, u, d = gu[:, :f].float(), gu[:, f:].float(), d2.float()
            sg = torch.sigmoid(g)
            grad = torch.cat([d * u * sg * (1 + g * (1 - sg)), d * g * sg], 1)
            return grad.to(gate_up.dtype).reshape(gate_up.shape)
        grad = torch.empty_like(gu)
        fn = _native.cuda().ka_swiglu_bwd
        _check(fn(gu.data_ptr(), gu.data_ptr() + 2 * f, 2 * f, d2.data_ptr(), grad.data_ptr(),
                  grad.data_ptr() + 2 * f, 2 * f, rows, f, _sms(gu), _stream(gu)), "ka_swiglu_bwd")
        return grad.reshape(gate_up.shape)


def swiglu_fn(gate_up: torch.Tensor) -> torch.Tensor:
    """Differentiable SwiGLU on a contiguous ``[..., 2F]`` tensor holding ``[gate | up]``."""
    if not gate_up.requires_grad or not torch.is_grad_enabled():
        return swiglu(gate_up)
    return _SwigluFn.apply(gate_up.contiguous())
