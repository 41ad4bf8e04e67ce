"""No kernel touches the shared memory of another CTA of its cluster before a cluster barrier: until then that CTA need
not have started. Read from the sources, in the order of the text, with calls of device functions followed."""
import os
import re

import pytest

FOLDER = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "csrc", "sm100")
WAIT = re.compile(r"barrier\.cluster\.wait")
REMOTE = re.compile(r"(?:ld|st|atom|red)\.(?:async\.)?shared::cluster|mbarrier\.arrive\.[\w:.]*shared::cluster")


def _read(name):
    """The file, behind the headers that all of them share, without comments."""
    common = os.path.join(FOLDER, "common")
    paths = [os.path.join(common, n) for n in sorted(os.listdir(common))] + \
        [os.path.join(FOLDER, n) for n in sorted(os.listdir(FOLDER)) if n.endswith(".cuh")] + [os.path.join(FOLDER, name)]
    text = ""
    for path in paths:
        with open(path) as f:
            text += re.sub(r"//[^\n]*", "", f.read())
    return text


def _block(text, at):
    """From the brace at or behind ``at`` to the one that closes it."""
    at = text.index("{", at)
    depth = 0
    for i in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[at:i + 1]
    raise AssertionError("no end")


def _functions(text):
    """Bodies by name, all overloads of a name one behind the other, and the kernels' names."""
    out, kernels = {}, []
    for m in re.finditer(r"__(device|global)__", text):
        head = re.match(r"[^;{]*", text[m.end():m.end() + 4000]).group(0)
        name = re.search(r"(\w+)\s*\(", re.sub(r"__(launch_bounds|cluster_dims)__\s*\([^)]*\)", "", head))
        if text[m.end() + len(head)] == ";" or name is None:
            continue
        out[name.group(1)] = out.get(name.group(1), "") + _block(text, m.end())
        if m.group(1) == "global":
            kernels.append(name.group(1))
    return out, kernels


def _first(name, functions, known):
    """'wait' or 'remote', whichever the function comes to first, or None."""
    if name not in known:
        known[name] = None             # while it is being looked at
        for m in re.finditer(r"%s|(?P<remote>%s)|(?P<call>\b\w+)(?=\s*(?:<[\w\s,:]*>)?\s*\()" % (WAIT.pattern, REMOTE.pattern),
                             functions[name]):
            call = m.group("call")
            found = ("remote" if m.group("remote") else "wait") if call is None else \
                _first(call, functions, known) if call in functions and call != name else None
            if found:
                known[name] = found
                break
    return known[name]


def _kernels(text):
    functions, kernels = _functions(text)
    known = {}
    return {k: _first(k, functions, known) for k in kernels}


SOURCES = sorted(n for n in os.listdir(FOLDER) if n.endswith(".cu"))


@pytest.mark.parametrize("name", SOURCES)
def test_no_remote_shared_memory_before_a_cluster_barrier(name):
    found = _kernels(_read(name))
    assert "remote" not in found.values(), found


def test_the_kernels_with_clusters_are_seen():
    found = {k: v for name in SOURCES for k, v in _kernels(_read(name)).items()}
    for kernel in ("sample_parts_kernel", "sample_topk_held_kernel", "attention_decode_split_kernel", "gemm_bf16_kernel"):
        assert found[kernel] == "wait", kernel
    bad = "__device__ void put(int a) { asm volatile(\"st.shared::cluster.u32 [%0], %1;\"); }\n" \
          "__device__ void wait() { asm volatile(\"barrier.cluster.wait.acquire;\"); }\n" \
          "__global__ void __launch_bounds__(kT, 1) k(int a) { __syncthreads(); put(a); wait(); }\n"
    assert _kernels(bad) == {"k": "remote"}
