"""Size rules of the CUDA sources, compiled for the host: the weight gradient's
split into CTAs (csrc/model.cuh) and the long rows' sort space (csrc/prep.cuh)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SPLIT = r"""
#include <algorithm>
#include <cstdio>
#include "model.cuh"
int main() {
  uint32_t most = 0;
  for (uint32_t b = 1; b <= 60000; ++b) {
    const uint32_t ctas = tb::wgrad_ctas(b), rows = tb::wgrad_rows(b);
    if (rows % tb::wgrad_unit(b) || (uint64_t)ctas * rows < b || ctas > tb::kGradCtas) return std::printf("split %u\n", b), 1;
    most = std::max(most, ctas);  // the most CTAs a batch of up to b rows takes
    if (tb::wgrad_parts(b) < most) return std::printf("%u rows: %u parts, %u CTAs\n", b, tb::wgrad_parts(b), most), 1;
  }
  for (uint32_t b : {1u << 20, 1u << 31, 0xFFFFFFFFu})
    if (tb::wgrad_parts(b) != tb::kGradCtas || tb::wgrad_ctas(b) > tb::kGradCtas) return std::printf("large %u\n", b), 1;
  return 0;
}
"""


SORT_SPACE = r"""
#include <cstdio>
#include "prep.cuh"
int main() {
  // The most entries, all in rows of one length that sorts in global scratch:
  // 8,193 entries are padded to 16,384 words.
  const uint32_t length = 8193, words = 16384;
  tb::SortSpace taken = 0;
  for (uint64_t entries = 0; entries + length <= tb::kMaxEntries; entries += length) {
    const tb::SortSpace at = taken;
    taken += words;
    if (taken <= at) return std::printf("a slice starts over at entry %llu\n", (unsigned long long)entries), 1;
  }
  return taken > 2 * tb::kMaxEntries;
}
"""


def _run(tmp_path, program):
    src, exe = tmp_path / "sizes.cu", str(tmp_path / "sizes")
    src.write_text(program)
    subprocess.run(["nvcc", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
                    "-I", os.path.join(ROOT, "tribit_b200", "csrc"), "-I", os.path.join(ROOT, "include"), "-o", exe,
                    str(src)], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_partial_sums_hold_every_shorter_batch(tmp_path):
    _run(tmp_path, SPLIT)


def test_sort_space_of_the_most_entries(tmp_path):
    _run(tmp_path, SORT_SPACE)
