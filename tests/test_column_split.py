"""Columns split over CTAs: the TMA-fed kernels divide a column's levels among CTAs by a rule
on the grid.  The rule has to cover every level once, and the split kernels have to give the
values of the overlapped-tile kernels, which march whole columns, bit for bit."""
import subprocess

import numpy as np
import pytest

from conftest import ROOT

SPLIT_MAIN = r"""
#include "zsplit.cuh"
#include <cstdio>
int main() {
  const int tiles[] = {1, 2, 12, 77, 128, 288, 425, 512, 2048, 9000};
  const float extra[] = {0.7f, 1.0f, 1.5f, 3.0f};
  for (int t : tiles)
    for (int nz = 1; nz <= 256; ++nz)
      for (int ctas = 2; ctas <= 4; ++ctas)
        for (float e : extra) {
          const gwmb::ZSplit s = gwmb::z_split_search(t, nz, 148 * ctas, e);
          int at = 0;
          for (int z = 0; z < s.chunks; ++z) {
            if (s.first(z) != at || s.last(z, nz) <= at || s.last(z, nz) - at > s.longest()) return 1;
            at = s.last(z, nz);
          }
          if (at != nz) return 2;
        }
  std::puts("ok");
  return 0;
}
"""


def test_split_covers_every_level_once(tmp_path):
    src = tmp_path / "split.cpp"
    src.write_text(SPLIT_MAIN)
    exe = tmp_path / "split"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", f"{ROOT}/gpu-wm-next_b200/csrc", "-I", "/usr/local/cuda/include",
                    "-o", str(exe), str(src), "-L", "/usr/local/cuda/lib64", "-lcudart",
                    "-Wl,-rpath,/usr/local/cuda/lib64"], check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.strip() == "ok"


# tile edges and remainders; one level, fewer levels than a chunk, chunks with a remainder;
# a grid wide enough for uneven chunks (700 x 340: 484 tiles)
SHAPES = [(32, 16, 1), (33, 17, 2), (31, 15, 3), (64, 32, 7), (65, 47, 41), (34, 250, 64), (700, 340, 21)]


@pytest.mark.gpu
@pytest.mark.parametrize("terrain", [False, True])
@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("nx,ny,nz", SHAPES)
def test_split_columns_match_whole_columns(gwm, nx, ny, nz, periodic, terrain):
    hill = None
    if terrain:
        hill = gwm.build_terrain("cosine_mountain", nx, ny, 1000.0, 1000.0, height=300.0, half_width_x=0.3,
                                 half_width_y=0.3)
    grid = gwm.GridSpec(nx, ny, nz, dx=1000.0, dy=1000.0, z_top=300.0 * nz, terrain=hill, periodic_x=periodic,
                        periodic_y=periodic)
    state = gwm.build_case("moist_sounding", gwm.GridSpec(nx, ny, nz, dx=1000.0, dy=1000.0, z_top=300.0 * nz),
                           gwm.CaseParams(theta_ref=300.0, noise_rms_k=0.5, seed=3, relative_humidity=1.01), moist=True)
    rng = np.random.default_rng(1)
    state["u"] = (state["u"] + rng.normal(2.0, 1.0, state["u"].shape)).astype(np.float32)
    state["u"][:, :, -1] = state["u"][:, :, 0]
    spec = gwm.MemberSpec(step=gwm.StepConfig(dt=0.5, fast_substeps=3),
                          rain=gwm.WarmRainConfig(dt=0.5, rain_terminal_velocity=12.0), moist=True)
    out = {}
    with gwm.Model(grid, spec) as m:
        for rows in (8, 3):
            for kernel in ("slow_stage", "fast_substep", "tracer_stage"):
                m.set_tile(kernel, rows)
            m.upload(dict(state, precip=np.zeros((ny, nx))))
            m.step(2)
            out[rows] = m.download()
    for k in out[3]:
        np.testing.assert_array_equal(out[3][k], out[8][k], err_msg=f"{k} of split columns")
