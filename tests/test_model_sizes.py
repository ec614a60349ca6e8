"""The weight gradient's split into CTAs (csrc/model.cuh), compiled for the host."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = r"""
#include <algorithm>
#include <cstdio>
#include "model.cuh"
int main() {
  uint32_t most = 0;
  for (uint32_t b = 1; b <= 60000; ++b) {
    const uint32_t ctas = tb::wgrad_ctas(b), rows = tb::wgrad_rows(b);
    if (rows % tb::kGradTile || (uint64_t)ctas * rows < b || ctas > tb::kGradCtas) return std::printf("split %u\n", b), 1;
    most = std::max(most, ctas);  // the most CTAs a batch of up to b rows takes
    if (tb::wgrad_parts(b) < most) return std::printf("%u rows: %u parts, %u CTAs\n", b, tb::wgrad_parts(b), most), 1;
  }
  for (uint32_t b : {1u << 20, 1u << 31, 0xFFFFFFFFu})
    if (tb::wgrad_parts(b) != tb::kGradCtas || tb::wgrad_ctas(b) > tb::kGradCtas) return std::printf("large %u\n", b), 1;
  return 0;
}
"""


def test_partial_sums_hold_every_shorter_batch(tmp_path):
    src = tmp_path / "sizes.cu"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "sizes")
    subprocess.run(["nvcc", "-std=c++17", "-I", os.path.join(ROOT, "tribit_b200", "csrc"), "-I",
                    os.path.join(ROOT, "include"), "-o", exe, str(src)], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
