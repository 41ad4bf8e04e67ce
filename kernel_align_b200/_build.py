"""Native build, in-tree: nvcc for the sm_100a kernels, g++ for the CPU oracle library and for the
operators that are C++ autograd nodes.

The first two are plain shared objects with ``extern "C"`` entry points, loaded through
``ctypes``, the third is an extension module against the installed torch; they sit next to the package so that a
built tree can be copied to a GPU host as is. A content hash of the sources and flags decides whether a rebuild is needed.
An installed package carries the built libraries and the sources of the third alone, which ``python -m kernel_align_b200._build``
compiles there if the package was built without a torch, or beside another one.
"""
from __future__ import annotations

import hashlib
import os
import shutil
import subprocess
import sys
import sysconfig
import threading
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "csrc"
LIB_DIR = Path(__file__).resolve().parent / "_lib"
OBJ_DIR = ROOT / "build" / "obj"

CUDA_LIB = LIB_DIR / "libka_sm100.so"
CPU_LIB = LIB_DIR / "libka_cpu.so"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
    "-diag-suppress", "177",
]
CXX_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-ffp-contract=off", "-fno-fast-math", "-pthread"]


def _nvcc() -> str | None:
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    return cand if os.path.exists(cand) else None


def _digest(files: list[Path], flags: list[str]) -> str:
    h = hashlib.sha256()
    h.update(" ".join(flags).encode())
    for f in sorted(files):
        h.update(str(f.relative_to(ROOT)).encode())
        h.update(f.read_bytes())
    return h.hexdigest()


def _run(cmd: list[str]) -> None:
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
        raise RuntimeError(f"native build failed: {' '.join(cmd[:3])} ...")


def _stamp_ok(lib: Path, digest: str) -> bool:
    stamp = lib.with_suffix(".hash")
    return lib.exists() and stamp.exists() and stamp.read_text().strip() == digest


def build_cuda(force: bool = False, verbose: bool = False) -> Path | None:
    """Compile every ``csrc/sm100/*.cu`` for sm_100a and link ``libka_sm100.so``."""
    nvcc = _nvcc()
    srcs = sorted((CSRC / "sm100").glob("*.cu"))
    if not srcs:      # an installed wheel carries the built library, not the sources
        return CUDA_LIB if CUDA_LIB.exists() else None
    deps = srcs + sorted((CSRC / "sm100").rglob("*.cuh")) + sorted((CSRC / "sm100").rglob("*.h"))
    digest = _digest(deps, NVCC_FLAGS)
    if not force and _stamp_ok(CUDA_LIB, digest):
        return CUDA_LIB
    if nvcc is None:
        return CUDA_LIB if CUDA_LIB.exists() else None
    LIB_DIR.mkdir(parents=True, exist_ok=True)
    OBJ_DIR.mkdir(parents=True, exist_ok=True)
    extra = ["-Xptxas", "-v"] if verbose else []

    def one(src: Path) -> Path:
        obj = OBJ_DIR / (src.stem + ".o")
        _run([nvcc, *NVCC_FLAGS, *extra, "-I", str(CSRC / "sm100"), "-c", str(src), "-o", str(obj)])
        return obj

    with ThreadPoolExecutor(max_workers=min(8, max(1, len(srcs)))) as ex:
        objs = list(ex.map(one, srcs))
    _run([nvcc, "-shared", "-o", str(CUDA_LIB), *[str(o) for o in objs], "-cudart", "static"])
    CUDA_LIB.with_suffix(".hash").write_text(digest)
    return CUDA_LIB


def build_cpu(force: bool = False) -> Path | None:
    """Compile ``csrc/cpu/*.cpp`` into ``libka_cpu.so`` (the CPU oracle and CPU code path)."""
    srcs = sorted((CSRC / "cpu").glob("*.cpp"))
    if not srcs:
        return CPU_LIB if CPU_LIB.exists() else None
    deps = srcs + sorted((CSRC / "cpu").rglob("*.h"))
    digest = _digest(deps, CXX_FLAGS)
    if not force and _stamp_ok(CPU_LIB, digest):
        return CPU_LIB
    cxx = shutil.which("g++")
    if cxx is None:
        return CPU_LIB if CPU_LIB.exists() else None
    LIB_DIR.mkdir(parents=True, exist_ok=True)
    _run([cxx, *CXX_FLAGS, "-shared", "-o", str(CPU_LIB), *[str(s) for s in srcs]])
    CPU_LIB.with_suffix(".hash").write_text(digest)
    return CPU_LIB


def torch_lib() -> Path | None:
    """Where the extension module for this Python and this torch is, or would be; None without torch. An extension of
    another torch must not be loaded, so both versions are part of its name: a package that was built beside
    another torch has none."""
    try:
        import torch
    except ImportError:
        return None
    return LIB_DIR / f"_ka_torch.cp{sys.version_info.major}{sys.version_info.minor}.torch{torch.__version__}.so"


def torch_missing() -> str | None:
    """Why the extension module cannot be compiled on this host, or None if it can."""
    try:
        import torch
    except ImportError:
        return "torch is not installed"
    if torch.version.cuda is None or not (Path(torch.__file__).parent / "lib" / "libc10_cuda.so").exists():
        return "this torch was built without CUDA"
    if _cuda_include() is None:
        return "no CUDA headers (cuda_runtime_api.h) under CUDA_HOME, beside nvcc or under /usr/local/cuda"
    if shutil.which("g++") is None:
        return "no g++"
    return None


def _cuda_include() -> Path | None:
    nvcc = _nvcc()
    homes = [os.environ.get("CUDA_HOME"), nvcc and Path(nvcc).resolve().parent.parent, "/usr/local/cuda"]
    for home in homes:
        if home and (Path(home) / "include" / "cuda_runtime_api.h").exists():
            return Path(home) / "include"
    return None


def build_torch(force: bool = False, installed: bool = False) -> Path | None:
    """Compile ``csrc/torch/*.cpp`` into the extension module ``_ka_torch.*.so`` (C++ autograd nodes). None where that is
    not possible (:func:`torch_missing`): the operators then reach the kernels from Python. An installed package compiles
    nothing unless ``installed`` is set: it takes the module that it was built with, if that is one for this torch."""
    out = torch_lib()
    if out is None:
        return None
    srcs = sorted((CSRC / "torch").glob("*.cpp"))
    if not srcs:
        if not installed or out.exists():
            return out if out.exists() else None
        srcs = sorted((LIB_DIR.parent / "_src").glob("*.cpp"))
        if not srcs:
            return None
    import torch

    inc, lib = Path(torch.__file__).parent / "include", Path(torch.__file__).parent / "lib"
    flags = ["-O2", "-std=c++17", "-fPIC", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}"]
    digest = _digest(srcs, [*flags, torch.__version__, sys.version])
    if not force and _stamp_ok(out, digest):
        return out
    if torch_missing() is not None:
        return None
    LIB_DIR.mkdir(parents=True, exist_ok=True)
    # ranks that build at the same time, at their first call, each find a whole file
    part = out.with_name(f"{out.stem}.{os.getpid()}.{threading.get_ident()}.part")
    try:
        _run(["g++", *flags, "-shared", "-o", str(part), *[str(s) for s in srcs], f"-I{inc}",
              f"-I{inc / 'torch' / 'csrc' / 'api' / 'include'}", f"-I{sysconfig.get_paths()['include']}",
              f"-I{_cuda_include()}", f"-L{lib}", "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda"])
        os.replace(part, out)
    except RuntimeError:     # the compiler's message is on stderr; the other libraries do not need this one
        return None
    finally:
        part.unlink(missing_ok=True)
    out.with_suffix(".hash").write_text(digest)
    return out


def build_cpu_sanitized(force: bool = False) -> Path | None:
    """The CPU library once more with AddressSanitizer and UndefinedBehaviorSanitizer
    (``libka_cpu_asan.so``): the sanitizer tier of the tests loads it in a child process that
    preloads the sanitizer runtime. Not used by the package itself."""
    srcs = sorted((CSRC / "cpu").glob("*.cpp"))
    cxx = shutil.which("g++")
    if not srcs or cxx is None:
        return None
    flags = [f for f in CXX_FLAGS if not f.startswith("-O")] + ["-O1", "-g", "-fno-omit-frame-pointer",
                                                                 "-fsanitize=address,undefined",
                                                                 "-fno-sanitize-recover=undefined"]
    deps = srcs + sorted((CSRC / "cpu").rglob("*.h"))
    digest = _digest(deps, flags)
    lib = LIB_DIR / "libka_cpu_asan.so"
    if not force and _stamp_ok(lib, digest):
        return lib
    LIB_DIR.mkdir(parents=True, exist_ok=True)
    _run([cxx, *flags, "-shared", "-o", str(lib), *[str(s) for s in srcs]])
    lib.with_suffix(".hash").write_text(digest)
    return lib


def sanitizer_runtime() -> str | None:
    """Path of the AddressSanitizer runtime to preload, or None without g++."""
    cxx = shutil.which("g++")
    if cxx is None:
        return None
    out = subprocess.run([cxx, "-print-file-name=libasan.so"], capture_output=True, text=True).stdout.strip()
    return out if out and os.path.exists(out) else None


def build_all(force: bool = False, verbose: bool = False) -> None:
    build_cpu(force)
    build_cuda(force, verbose)
    build_torch(force, installed=True)


if __name__ == "__main__":
    build_all(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print("built:", [str(p) for p in (CPU_LIB, torch_lib(), CUDA_LIB) if p is not None and p.exists()])
