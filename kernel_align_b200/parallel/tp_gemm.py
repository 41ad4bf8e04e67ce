"""Tensor-parallel linear layers whose collective runs inside the GEMM kernel.

``gemm_reduce_scatter(x, w_shard, ctx)``: row-parallel linear (``x [M, K/world]``,
``w_shard [N, K/world]``) -> this rank's rows ``[M/world, N]`` of ``x_full @ w_full.T`` (+ residual).
``all_gather_gemm(x_local, w_shard, ctx)``: column-parallel linear on row-sharded input
(``x_local [M/world, K]``, ``w_shard [N/world, K]``) -> ``[M, N/world]``.

Kernels: ``csrc/sm100/tp_gemm.cu`` / ``gemm.cu``; peer buffers: :class:`PeerArena`. With
``world == 1`` the same kernels run on local buffers, which is what makes TP=1 and TP=8 agree
bit for bit: K is always reduced as 8 canonical slices in one fixed tree order.

CPU tensors take a PyTorch path with the same arithmetic contract (8 canonical K slices, each
partial rounded to bf16, the fixed tree, residual added after rounding), exchanging over the
process group's CPU backend (gloo): it is what the multi-process CPU tests run, and it is
invariant in the number of ranks for the same reason the kernels are.
"""
from __future__ import annotations

from ctypes import c_void_p
from typing import Optional

import torch
import torch.distributed as dist

from .. import _native
from ..ops.fused_logp import default_timeout_ns
from ..ops.gemm import status_buffer
from ..utils.profiler import profiled


class _LocalArena:
    """Stand-in for :class:`PeerArena` when there is a single rank."""

    def __init__(self, nbytes: int, device):
        self.buf = torch.zeros(nbytes, dtype=torch.uint8, device=device)
        self.ptrs = [self.buf.data_ptr()]
        self.rank, self.world = 0, 1


class TPContext:
    """Process-group handle plus the exchange buffers of the fused TP kernels (allocated on
    first use per shape, then reused; each buffer carries its own call counter)."""

    def __init__(self, group: Optional[dist.ProcessGroup] = None, device=None):
        if dist.is_available() and dist.is_initialized():
            self.group = group if group is not None else dist.group.WORLD
            self.rank = dist.get_rank(self.group)
            self.world = dist.get_world_size(self.group)
        else:
            self.group, self.rank, self.world = None, 0, 1
        if device is not None:
            self.device = torch.device(device)
        elif torch.cuda.is_available():
            self.device = torch.device("cuda", torch.cuda.current_device())
        else:
            self.device = torch.device("cpu")
        self._arenas: dict = {}

    def arena(self, key, nbytes: int):
        ent = self._arenas.get(key)
        if ent is None:
            if self.world == 1:
                ar = _LocalArena(nbytes, self.device)
            else:
                from .peer import PeerArena

                ar = PeerArena(nbytes, self.group, self.device)
            ent = [ar, 0]
            self._arenas[key] = ent
        ent[1] += 1
        return ent[0], ent[1]


def _tree8(p: torch.Tensor) -> torch.Tensor:
    """``p [8, ...]`` fp32 -> ((0+1)+(2+3))+((4+5)+(6+7))."""
    return ((p[0] + p[1]) + (p[2] + p[3])) + ((p[4] + p[5]) + (p[6] + p[7]))


def _gemm_reduce_scatter_cpu(x, w_shard, ctx, residual, trans_b, keep_padding):
    m, k_local = x.shape
    wf = w_shard.float().t() if trans_b else w_shard.float()          # [N, K_local]
    n = wf.shape[0]
    s_local = 8 // ctx.world
    ks = k_local // s_local
    xf = x.float()
    from ..ops import cpu_ops

    parts = torch.stack([cpu_ops.gemm_cpu(xf[:, i * ks:(i + 1) * ks].contiguous(),
                                          wf[:, i * ks:(i + 1) * ks].contiguous()).to(torch.bfloat16).float()
                         for i in range(s_local)])                       # this rank's slices, rounded
    if ctx.world > 1:
        gathered = [torch.empty_like(parts) for _ in range(ctx.world)]
        dist.all_gather(gathered, parts.contiguous(), group=ctx.group)
        parts = torch.cat(gathered)
    v = _tree8(parts)
    rpr = rows_per_rank(m, ctx.world)
    lo = ctx.rank * rpr
    rows_valid = max(0, min(rpr, m - lo))
    out = torch.zeros(rpr, n, dtype=torch.float32)
    out[:rows_valid] = v[lo:lo + rows_valid]
    if residual is not None:
        res = residual.float()
        if res.shape[0] < rpr:
            res = torch.cat([res, res.new_zeros(rpr - res.shape[0], n)])
        out = out.to(torch.bfloat16).float() + res[:rpr]
    out = out.to(torch.bfloat16)
    return out if keep_padding else out[:rows_valid]


def _split_pays(m: int, n: int, k: int) -> bool:
    """Whether one rank that sums its eight K slices itself makes them units of their own
    (``ka_gemm_split8``: eight times as many units, a pass over the partials) or keeps a tile's slices on one
    CTA pair (``ka_gemm_tree8``). Measured split / kept in us on 74 pairs, calls after one another (19 us is what
    the host takes for one, so K = 1024 tells little), tiles counted as 256 x 256: 16 tiles: 27 / 34 (K = 4096),
    34 / 83 (14336), 55 / 153 (28672); 24 tiles: 21 / 20 (1024), 26 / 34 (4096), 47 / 84 (14336); 32 tiles: 23 / 20
    (1024), 29 / 34 (4096), 58 / 86 (14336), 103 / 157 (28672); 48 tiles: 33 / 32 (1024), 44 / 46 (4096), 51 / 56
    (6144), 85 / 99 (14336), 148 / 175 (28672); 64 tiles: 39 / 32 (1024), 53 / 49 (4096), 63 / 60 (6144), 102 / 105
    (14336), 180 / 188 (28672). One row instead, whose tiles are mostly padding: 20 tiles 25 / 34 (4096),
    83 / 157 (28672); 32 tiles 29 / 38, 107 / 171. With more tiles the partials outgrow what the rest saves, with half a
    gigabyte of scratch at 256 of them."""
    tiles = -(-m // 256) * -(-n // 256)
    return tiles <= 24 or (tiles <= 48 and k >= 4096) or (tiles <= 64 and k >= 12288)


def _tree_pays(m: int, n: int, k: int, num_sms: int) -> bool:
    """Whether one rank sums its eight K slices itself, in one of the two forms of :func:`_split_pays`, or
    stages them as several ranks do (``ka_gemm_reduce_scatter``). The bits are the same.

    Staged slices spread over all pairs but cost fences, flags and the wait for them. Measured on
    148 SMs, staged / own in us, tiles counted as 256 x 256: 256 tiles: 385 / 156 (K = 4096; 139 since TMEM is
    handed back without waiting for stores), 1025 / 738 (28672);
    32 tiles: 72 / 32 (4096), 109 / 61 (14336), 150 / 101 (28672); 16 tiles: 48 / 20 (4096), 57 / 24 (6144),
    70 / 37 (14336), 101 / 58 (28672); 4 tiles: 39 / 19 (4096). A slice round of a kept tile takes about 5.4e-3 us
    per K column, staging about 20 us plus 1.2 us per tile; the rule compares the two."""
    if _split_pays(m, n, k):
        return True
    pairs = max(1, num_sms // 2)
    tiles = -(-m // 256) * -(-n // 256)
    extra_rounds = -(-tiles // pairs) * 8 - -(-8 * tiles // pairs)
    return extra_rounds * (k / 8) * 5.4e-3 < 20 + 1.2 * tiles


@profiled("gemm_reduce_scatter")
def gemm_reduce_scatter(x: torch.Tensor, w_shard: torch.Tensor, ctx: TPContext,
                        residual: Optional[torch.Tensor] = None, trans_b: bool = False,
                        keep_padding: bool = False) -> torch.Tensor:
    """Rows ``[rank * M/world, (rank + 1) * M/world)`` of ``concat_k(x) @ concat_k(w).T`` (+ residual).

    ``w_shard`` is ``[N, K_local]``, or ``[K_local, N]`` with ``trans_b``. ``keep_padding`` returns
    all ``rows_per_rank`` rows (a multiple of 128) instead of cutting at the end of the matrix."""
    m, k_local = x.shape
    n = w_shard.shape[1] if trans_b else w_shard.shape[0]
    if k_local % (8 // ctx.world * 64) != 0:
        raise ValueError("the K shard must split into whole 64-wide blocks per canonical slice")
    if x.device.type != "cuda":
        return _gemm_reduce_scatter_cpu(x, w_shard, ctx, residual, trans_b, keep_padding)
    lib = _native.cuda()
    x = x.contiguous()
    w = w_shard.contiguous()
    rpr = rows_per_rank(m, ctx.world)
    rows_valid = max(0, min(rpr, m - ctx.rank * rpr))
    out = torch.empty(rpr, n, dtype=torch.bfloat16, device=x.device)
    res = None
    if residual is not None:
        res = residual.contiguous()
        if res.shape[0] < rpr:
            res = torch.cat([res, res.new_zeros(rpr - res.shape[0], n)])
        elif res.data_ptr() % 16:
            res = res.clone()
    sms = _native.sm_count(x.device)
    if ctx.world == 1 and _tree_pays(m, n, k_local, sms):
        if _split_pays(m, n, k_local):
            scratch = torch.empty(lib.ka_gemm_split8_scratch_elems(m, n), dtype=torch.bfloat16, device=x.device)
            fn = lib.ka_gemm_split8
        else:
            scratch = torch.empty(lib.ka_gemm_tree8_scratch_bytes(sms), dtype=torch.uint8, device=x.device)
            fn = lib.ka_gemm_tree8
        rc = fn(x.data_ptr(), x.stride(0), w.data_ptr(), w.stride(0), int(trans_b), out.data_ptr(),
                res.data_ptr() if res is not None else None, scratch.data_ptr(), m, n, k_local,
                status_buffer(x.device).data_ptr(), sms, default_timeout_ns(), _native.stream_ptr(x.device))
        if rc != 0:
            raise RuntimeError(f"the row-parallel product rejected its arguments (code {rc})")
        return out if keep_padding else out[:rows_valid]
    nbytes = lib.ka_gemm_rs_exchange_bytes(m, n, ctx.world)
    arena, epoch = ctx.arena(("rs", m, n), nbytes)
    ptrs = (c_void_p * ctx.world)(*arena.ptrs)
    rc = lib.ka_gemm_reduce_scatter(x.data_ptr(), x.stride(0), w.data_ptr(), w.stride(0), int(trans_b), out.data_ptr(),
                                    res.data_ptr() if res is not None else None, ptrs, m, n, k_local, ctx.world,
                                    ctx.rank, epoch & 0xFFFFFFFF, status_buffer(x.device).data_ptr(),
                                    sms, default_timeout_ns(), _native.stream_ptr(x.device))
    if rc != 0:
        raise RuntimeError(f"ka_gemm_reduce_scatter rejected its arguments (code {rc})")
    return out if keep_padding else out[:rows_valid]


def rows_per_rank(m: int, world: int) -> int:
    """Rows of a reduce-scattered ``[m, n]`` result that each rank owns (multiple of 128; the
    same rule as ``ka_gemm_rs_rows_per_rank``)."""
    per = (m + world - 1) // world
    return (per + 127) // 128 * 128


@profiled("all_gather_gemm")
def all_gather_gemm(x_local: torch.Tensor, w_shard: torch.Tensor, ctx: TPContext, trans_b: bool = False,
                    return_gathered: bool = False):
    """``all_gather(x_local, dim=0) @ w_shard.T``; ``x_local`` rows must be a multiple of 128.

    ``w_shard`` is ``[N_local, K]``, or ``[K, N_local]`` with ``trans_b``. With ``return_gathered``
    also returns a copy of the gathered activations ``[world * rows, K]``."""
    rows, k = x_local.shape
    n_local = w_shard.shape[1] if trans_b else w_shard.shape[0]
    if rows % 128 != 0:
        raise ValueError("rows per rank must be a multiple of 128")
    if x_local.device.type != "cuda":
        from ..ops.gemm import gemm_bi

        if ctx.world > 1:
            pieces = [torch.empty_like(x_local) for _ in range(ctx.world)]
            dist.all_gather(pieces, x_local.contiguous(), group=ctx.group)
            x_full = torch.cat(pieces)
        else:
            x_full = x_local
        out = gemm_bi(x_full, w_shard, trans_b=trans_b)
        return (out, x_full.clone()) if return_gathered else out
    lib = _native.cuda()
    x = x_local.contiguous()
    w = w_shard.contiguous()
    nbytes = lib.ka_ag_gemm_exchange_bytes(rows, k, ctx.world)
    arena, epoch = ctx.arena(("ag", rows, k), nbytes)
    out = torch.empty(ctx.world * rows, n_local, dtype=torch.bfloat16, device=x.device)
    ptrs = (c_void_p * ctx.world)(*arena.ptrs)
    sms = _native.sm_count(x.device)
    rc = lib.ka_all_gather_gemm(x.data_ptr(), w.data_ptr(), w.stride(0), int(trans_b), out.data_ptr(), out.stride(0), ptrs, rows,
                                n_local, k, ctx.world, ctx.rank, epoch & 0xFFFFFFFF,
                                status_buffer(x.device).data_ptr(), sms, default_timeout_ns(), _native.stream_ptr(x.device))
    if rc != 0:
        raise RuntimeError(f"ka_all_gather_gemm rejected its arguments (code {rc})")
    if return_gathered:
        nb = (ctx.world * rows * k * 2 + 255) // 256 * 256
        gen = epoch & 1
        gathered = arena.buf[gen * nb: gen * nb + ctx.world * rows * k * 2].view(torch.bfloat16).view(ctx.world * rows, k)
        return out, gathered.clone()
    return out
