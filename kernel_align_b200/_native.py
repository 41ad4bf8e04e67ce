"""Bindings to the in-tree native libraries: ctypes for two, an extension module for the third.

``cuda()`` returns the sm_100a kernel library and raises if it is missing: on a GPU host the
hand-written kernels are the only code path, there is no silent PyTorch fallback.
``cpu()`` returns the C++ CPU library (oracle for the tests and the CPU device path).
``torch_ops()`` returns the extension module with the operators that are C++ autograd nodes, or None: it is
made for one torch, which an isolated package build does not have, and the operators then reach the same kernels
through ``cuda()``.
"""
from __future__ import annotations

import ctypes
import importlib.util
import os
from ctypes import c_char_p, c_float, c_int, c_longlong, c_size_t, c_uint, c_ulonglong, c_void_p
from functools import lru_cache

from . import _build


class NativeLibraryMissing(RuntimeError):
    pass


def _bind(lib, name, restype, argtypes):
    fn = getattr(lib, name)
    fn.restype = restype
    fn.argtypes = argtypes
    return fn


@lru_cache(maxsize=None)
def cuda() -> ctypes.CDLL:
    path = _build.build_cuda()
    if path is None or not path.exists():
        raise NativeLibraryMissing(
            "libka_sm100.so is not built; run `python -m kernel_align_b200._build` on a host with nvcc"
        )
    lib = ctypes.CDLL(str(path))
    _bind(lib, "ka_lmhead_logp_workspace_bytes", c_size_t, [c_int, c_int])
    _bind(lib, "ka_lmhead_logp_status_offset", c_int, [c_int, c_int])
    _bind(lib, "ka_lmhead_logp_exchange_bytes", c_size_t, [c_int, c_int])
    _bind(
        lib,
        "ka_lmhead_logp_forward",
        c_int,
        [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_size_t, c_void_p,
         c_int, c_int, c_int, c_int, c_int, c_int, c_int,
         c_uint, c_float, c_int, c_int, c_int, c_ulonglong, c_void_p],
    )
    _bind(
        lib,
        "ka_lmhead_logp_forward_sched",
        c_int,
        [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_size_t, c_void_p,
         c_int, c_int, c_int, c_int, c_int, c_int, c_int,
         c_uint, c_float, c_int, c_int, c_int, c_int, c_int, c_int, c_ulonglong, c_void_p],
    )
    _bind(lib, "ka_lmhead_logp_gather_bytes", c_size_t, [c_int, c_int, c_int])
    _bind(
        lib,
        "ka_lmhead_logp_forward_sharded",
        c_int,
        [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_size_t, c_void_p, c_void_p,
         c_int, c_int, c_int, c_int, c_int, c_int, c_int,
         c_uint, c_float, c_int, c_int, c_int, c_int, c_int, c_int, c_int, c_ulonglong, c_void_p],
    )
    _bind(
        lib,
        "ka_sample",
        c_int,
        [c_void_p, c_int, c_longlong, c_int, c_int, c_void_p, c_float, c_int, c_float,
         c_ulonglong, c_ulonglong, c_void_p, c_void_p],
    )
    _bind(
        lib,
        "ka_logits_logp",
        c_int,
        [c_void_p, c_int, c_longlong, c_int, c_int, c_void_p, c_float, c_void_p, c_void_p, c_int, c_void_p],
    )
    _bind(lib, "ka_grpo_advantages", c_int, [c_void_p, c_void_p, c_int, c_int, c_float, c_void_p])
    _bind(
        lib,
        "ka_grpo_loss_fwd",
        c_int,
        [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_float, c_float, c_float, c_int,
         c_void_p, c_void_p, c_void_p, c_void_p, c_void_p],
    )
    _bind(lib, "ka_grpo_loss_bwd", c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_void_p])
    # prototypes are set here, once: setting them costs a call several microseconds
    p, i, ll, f, ull = c_void_p, c_int, c_longlong, c_float, c_ulonglong
    _bind(lib, "ka_rmsnorm", c_int, [p, p, p, p, p, i, i, f, i, p])
    _bind(lib, "ka_rmsnorm_bwd", c_int, [p, p, p, p, p, p, p, i, i, f, p])
    _bind(lib, "ka_rope", c_int, [p, ll, p, p, p, i, i, i, i, p])
    _bind(lib, "ka_qkv_rope", c_int, [p, ll, i, p, p, p, p, p, p, i, i, i, i, i, p])
    _bind(lib, "ka_swiglu", c_int, [p, p, ll, p, i, i, i, p])
    _bind(lib, "ka_swiglu_bwd", c_int, [p, p, ll, p, p, p, ll, i, i, i, p])
    _bind(lib, "ka_attention_fwd", c_int, [p, ll, p, ll, p, ll, p, ll, p, i, i, i, i, i, f, i, p, ull, p])
    _bind(lib, "ka_attention_bwd", c_int,
          [p, ll, p, ll, p, ll, p, ll, p, ll, p, p, p, ll, p, ll, p, ll, i, i, i, i, i, f, i, p, ull, p])
    _bind(lib, "ka_attention_decode", c_int, [p, p, p, p, p, i, i, i, i, i, f, p])
    _bind(lib, "ka_decode_qkv_rope_cache", c_int, [p, ll, p, p, p, p, p, p, p, i, i, i, i, p])
    _bind(lib, "ka_adamw_step", c_int, [p, p, p, i, p, p, ll, f, f, f, f, f, i, f, i, p])
    _bind(lib, "ka_gemm_bf16", c_int, [p, ll, i, p, ll, i, p, ll, i, i, i, i, p, i, ull, p])
    _bind(lib, "ka_gemm_skinny_bf16", c_int, [p, ll, p, ll, p, ll, i, i, i, p, ull, p])
    _bind(lib, "ka_lmhead_logits_grad", c_int, [p, p, p, p, p, p, ll, i, i, i, f, i, p, i, ull, p])
    _bind(lib, "ka_lmhead_kept_logits_grad", c_int, [p, p, p, p, p, i, i, f, p])
    _bind(lib, "ka_lmhead_logp_forward_keep", c_int,
          [p, p, p, p, p, p, p, c_size_t, i, i, i, c_uint, f, i, i, i, i, i, i, ull, p])
    _bind(lib, "ka_gemm_rs_exchange_bytes", c_size_t, [i, i, i])
    _bind(lib, "ka_gemm_rs_rows_per_rank", c_int, [i, i])
    _bind(lib, "ka_ag_gemm_exchange_bytes", c_size_t, [i, i, i])
    _bind(lib, "ka_gemm_reduce_scatter", c_int, [p, ll, p, ll, i, p, p, p, i, i, i, i, i, c_uint, p, i, ull, p])
    _bind(lib, "ka_gemm_tree8_scratch_bytes", c_size_t, [i])
    _bind(lib, "ka_gemm_tree8", c_int, [p, ll, p, ll, i, p, p, p, i, i, i, p, i, ull, p])
    _bind(lib, "ka_gemm_split8_scratch_elems", c_size_t, [i, i])
    _bind(lib, "ka_gemm_split8", c_int, [p, ll, p, ll, i, p, p, p, i, i, i, p, i, ull, p])
    _bind(lib, "ka_all_gather_gemm", c_int, [p, p, ll, i, p, ll, p, i, i, i, i, i, c_uint, p, i, ull, p])
    return lib


@lru_cache(maxsize=None)
def torch_ops():
    """The extension module with the operators that are C++ autograd nodes, bound to the kernels of :func:`cuda`; None
    if there is none for this torch and it cannot be built."""
    path = _build.build_torch()
    if path is None:
        return None
    spec = importlib.util.spec_from_file_location("_ka_torch", str(path))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    lib = cuda()
    mod.bind(*[ctypes.cast(getattr(lib, name), c_void_p).value
               for name in ("ka_grpo_advantages", "ka_grpo_loss_fwd", "ka_grpo_loss_bwd")])
    return mod


def _device_index(device) -> int:
    import torch

    return device.index if device.index is not None else torch.cuda.current_device()


def stream_ptr(device) -> int:
    """The current stream of a CUDA device as the integer the kernels take."""
    import torch

    return torch._C._cuda_getCurrentRawStream(_device_index(device))


@lru_cache(maxsize=None)
def _sm_count(index: int) -> int:
    import torch

    return torch.cuda.get_device_properties(index).multi_processor_count


def sm_count(device) -> int:
    """SMs of a CUDA device (asked once per device ordinal)."""
    return _sm_count(_device_index(device))


DTYPE_CODES = {"torch.float32": 0, "torch.bfloat16": 1, "torch.float16": 2}


def dtype_code(dtype) -> int:
    try:
        return DTYPE_CODES[str(dtype)]
    except KeyError:
        raise TypeError(f"unsupported dtype {dtype}; expected float32, bfloat16 or float16") from None


@lru_cache(maxsize=None)
def cpu() -> ctypes.CDLL:
    # KA_CPU_LIB points the process at another build of the same library (the sanitizer tier
    # of the tests runs the CPU operators on an ASan / UBSan build in a child process)
    override = os.environ.get("KA_CPU_LIB")
    if override:
        return ctypes.CDLL(override)
    path = _build.build_cpu()
    if path is None or not path.exists():
        raise NativeLibraryMissing("libka_cpu.so is not built and no C++ compiler is available")
    return ctypes.CDLL(str(path))


def cuda_available() -> bool:
    import torch

    return torch.cuda.is_available()
