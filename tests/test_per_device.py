"""Launch settings are kept per device (host logic, compiled with the host compiler), and a second GPU
of a process gets its own (two GPUs)."""
import os
import shutil
import subprocess

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

MAIN = r"""
#include <cassert>
#include <cstdio>
#include <thread>
#include <vector>
#include "common/per_device.h"
int main() {
  ka::PerDevice once, other;
  int calls = 0;
  auto ok = [&] { return 100 + ++calls; };
  assert(once.get(0, ok) == 101 && once.get(0, ok) == 101);       // set up once ...
  assert(once.get(1, ok) == 102 && once.get(0, ok) == 101);       // ... for every device
  assert(other.get(0, ok) == 103);                                // and for every kernel
  assert(once.get(2, [] { return -7; }) == -7 && once.get(2, ok) == 104);   // a failure is tried again
  assert(once.get(-1, ok) == -1 && once.get(64, ok) == -1 && calls == 4);
  std::vector<std::thread> threads;
  ka::PerDevice shared;
  int set_up = 0;                                                 // guarded by the object itself
  for (int t = 0; t < 8; ++t)
    threads.emplace_back([&] {
      for (int d = 0; d < 64; ++d) assert(shared.get(d, [&] { ++set_up; return d + 1; }) == d + 1);
    });
  for (auto& t : threads) t.join();
  assert(set_up == 64);
  std::puts("OK");
}
"""


def test_a_setting_is_made_once_per_device(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    src, exe = tmp_path / "main.cpp", tmp_path / "main"
    src.write_text(MAIN)
    subprocess.run([cxx, "-std=c++17", "-pthread", "-I", os.path.join(ROOT, "csrc", "sm100"), str(src), "-o", str(exe)],
                   check=True, timeout=120)
    assert subprocess.run([str(exe)], capture_output=True, text=True, timeout=60).stdout == "OK\n"


def test_no_launcher_keeps_a_setting_for_the_whole_process():
    """Every opt-in to shared memory is made on each call, or once per device."""
    folder = os.path.join(ROOT, "csrc", "sm100")
    for name in sorted(os.listdir(folder)):
        if name.endswith(".cu"):
            with open(os.path.join(folder, name)) as f:
                text = f.read()
            assert "static bool" not in text and "static int cached = " not in text, name


@pytest.mark.gpu
def test_gpu_a_second_device_takes_the_same_kernels(cuda_device):
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    from kernel_align_b200.ops.attention import attention_fn
    from kernel_align_b200.ops.gemm import gemm_bi
    from kernel_align_b200.ops.sampling import sample

    outs = []
    for dev in ("cuda:0", "cuda:1"):
        with torch.cuda.device(dev):
            g = torch.Generator().manual_seed(0)
            logits = (torch.randn(4, 50257, generator=g) * 2).half().to(dev)
            toks = [sample(logits, top_p=0.9, seed=1), sample(logits, top_k=50, seed=1), sample(logits.float(), top_k=50, seed=1)]
            x = torch.randn(300, 512, generator=g).bfloat16().to(dev)
            q, k, v = (torch.randn(1, 200, h, 128, generator=g).bfloat16().to(dev).requires_grad_() for h in (4, 2, 2))
            out = attention_fn(q, k, v)
            grads = torch.autograd.grad(out.float().sum(), (q, k, v))
            outs.append([t.cpu() for t in (*toks, gemm_bi(x, x[:128]), out, *grads)])
    assert all(torch.equal(a, b) for a, b in zip(*outs))
