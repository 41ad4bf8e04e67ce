"""Which 64 binades of a bf16 row the sampler counts (host arithmetic of ``sampling.cu``, compiled with the host compiler):
the ones that the row's maximum asks for serve every row, whatever the temperature."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

MAIN = r"""
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <vector>
#include "common/detmath.h"
using namespace ka;
using std::min;
#define __device__
#define __forceinline__ inline
static uint32_t __float_as_uint(float f) { return float_to_bits(f); }
static float __uint_as_float(uint32_t u) { return bits_to_float(u); }
%s
int main() {
  std::vector<float> inv_temps{INFINITY};
  for (int e = -149; e < 128; ++e)
    for (float m : {1.f, 1.37f}) inv_temps.push_back(std::ldexp(m, e));
  long rows = 0, bad = 0;
  for (float inv_temp : inv_temps)
    for (uint32_t bits = 0; bits < 65536; bits += 3) {
      const float x = bits16_float(bits), y_max = mul_rn(x, inv_temp);
      if (!std::isfinite(x) || !std::isfinite(y_max)) continue;
      const uint32_t mag = bits & 0x7FFFu, base = part_base(part_reach(x, inv_temp));
      const float lowest = -bits16_float(base + kPartMags);
      ++rows;
      const bool low = mass_fixed(exp_det(sub_rn(mul_rn(lowest, inv_temp), y_max))) != 0;
      if (base < 1 || base + kPartMags > 0x7F80 || mag >= base + kPartMags || low || !part_small_alike(base, inv_temp, y_max)) ++bad;
      // what counts as alike weighs alike
      for (uint32_t b : {base - 1, base / 2, 1u})
        for (uint32_t sign : {0u, 0x8000u})
          if (b < base && mass_fixed(exp_det(sub_rn(mul_rn(bits16_float(b | sign), inv_temp), y_max))) !=
                              mass_fixed(exp_det(sub_rn(0.f, y_max))))
            ++bad;
    }
  // with the binades that are counted at first: either alike, or counted again
  for (float inv_temp : inv_temps)
    for (uint32_t bits = 0; bits < 65536; bits += 7) {
      const float y_max = mul_rn(bits16_float(bits), inv_temp);
      if (!std::isfinite(y_max) || !part_small_alike(kPartBase, inv_temp, y_max)) continue;
      for (uint32_t b : {1u, 0x80u, 0x1234u, kPartBase - 1u})
        for (uint32_t sign : {0u, 0x8000u})
          if (mass_fixed(exp_det(sub_rn(mul_rn(bits16_float(b | sign), inv_temp), y_max))) !=
              mass_fixed(exp_det(sub_rn(0.f, y_max))))
            ++bad;
    }
  std::printf("%%ld %%ld\n", rows, bad);
}
"""


def test_the_binades_of_the_maximum_serve_every_row(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    with open(os.path.join(ROOT, "csrc", "sm100", "sampling.cu")) as f:
        text = f.read()
    parts = re.findall(r"constexpr int kPart(?:Binades|Mags|Base) = [^\n]*\n", text)
    for name in ("bits16_float", "part_reach", "part_base", "part_small_alike"):
        parts.append(re.search(r"__device__ __forceinline__ \w+ %s\(.*?\n?}\n" % name, text, re.S).group(0))
    assert len(parts) == 7
    src, exe = tmp_path / "main.cpp", tmp_path / "main"
    src.write_text(MAIN % "".join(parts))
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "csrc"), str(src), "-o", str(exe)],
                   check=True, timeout=120)
    rows, bad = map(int, subprocess.run([str(exe)], capture_output=True, text=True, timeout=300, check=True).stdout.split())
    assert rows > 1e7 and bad == 0, (rows, bad)
