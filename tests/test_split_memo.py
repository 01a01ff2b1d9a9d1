"""The splits that an ensemble's launches ask for, again and again, are searched for once."""
import subprocess

from conftest import ROOT

MEMO_MAIN = r"""
#include "zsplit.cuh"
#include <cstdio>
int main() {
  gwmb::SplitMemo memo;
  // the mixed members of an ensemble, and the (CTAs per SM, extra) of each kernel
  const int sizes[8][2] = {{6, 40}, {15, 64}, {24, 80}, {35, 40}, {54, 64}, {77, 80}, {104, 40}, {135, 64}};
  const struct { int ctas; float extra; } kernels[] = {{4, 0.7f}, {3, 1.0f}, {2, 1.0f}, {2, 1.2f}, {2, 1.5f}};
  for (int step = 0; step < 50; ++step)
    for (auto& m : sizes)
      for (auto& k : kernels) {
        const gwmb::ZSplit a = memo.get(m[0], m[1], 148 * k.ctas, k.extra);
        const gwmb::ZSplit b = gwmb::z_split_search(m[0], m[1], 148 * k.ctas, k.extra);
        if (a.big != b.big || a.nbig != b.nbig || a.small != b.small || a.chunks != b.chunks) return 1;
      }
  std::printf("%u\n", memo.searches);
  // more shapes than it holds: still the rule's answers
  for (int tiles = 1; tiles < 2000; ++tiles) {
    const gwmb::ZSplit a = memo.get(tiles, 1 + tiles % 256, 592, 0.7f);
    const gwmb::ZSplit b = gwmb::z_split_search(tiles, 1 + tiles % 256, 592, 0.7f);
    if (a.big != b.big || a.nbig != b.nbig || a.small != b.small || a.chunks != b.chunks) return 1;
  }
  return 0;
}
"""


def test_splits_of_mixed_members_are_searched_once(tmp_path):
    src = tmp_path / "memo.cpp"
    src.write_text(MEMO_MAIN)
    exe = tmp_path / "memo"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", f"{ROOT}/gpu-wm-next_b200/csrc", "-I", "/usr/local/cuda/include",
                    "-o", str(exe), str(src), "-L", "/usr/local/cuda/lib64", "-lcudart",
                    "-Wl,-rpath,/usr/local/cuda/lib64"], check=True)
    r = subprocess.run([str(exe)], check=True, capture_output=True, text=True)
    assert int(r.stdout) == 8 * 5
