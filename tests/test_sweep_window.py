"""The staged-record windows of the sparse-row sweeps, walked on the host with the functions the kernel
uses (sweep.cuh): whatever the row lengths, every record a lane reads lies inside its warp's own staging
buffer, and over the windows each row's records are read once."""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent / "dogpup_b200" / "csrc"

PROGRAM = r"""
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "sweep.cuh"
using namespace dgp::sweep;

template <class R> int walk(const std::vector<int> &rp, int nsp) {
  const int n = (int)rp.size() - 1, vec = nsp <= 8 ? 2 : 4;
  const Geo g = make_geo<R>(n, 1, nsp, vec, rp[n]);
  if (g.cap % 4 || stage_bytes<R>(g) > STAGE_MAX || stage_bytes<R>(g) < (size_t)WARPS * 2 * g.cap * Tr<R>::REC) return 1;
  for (int step = 0; step < g.steps; ++step)
    for (int warp = 0; warp < WARPS; ++warp) {
      const int r0 = (step * WARPS + warp) * g.rpw;
      auto bound = [&](int r) { return rp[std::min(r0 + std::min(r, g.rpw), n)]; };
      const int p0 = bound(0), pe = bound(g.rpw);
      std::vector<int> next(33);
      for (int r = 0; r <= g.rpw; ++r) next[r] = bound(r);
      // a lane's row and records: one lane per row leaves lanes 16.. for the rows' second halves
      const bool split = g.lpr == 1;
      struct Window {
        int first, count;
      };
      auto lane_window = [&](int lane, int c0) {
        const int r = split ? lane % 16 : lane / g.lpr;
        int b = bound(r), e = bound(r + 1);
        if (split) half_row(b, e, lane >= 16);
        Window w;
        w.first = window_first(b, c0);
        w.count = window_count(e, c0, g.cap, w.first, r < g.rpw && r0 + r < n);
        return w;
      };
      std::vector<char> seen(pe - p0 + 1, 0);
      for (int c0 = p0;;) {
        int m = 0;
        for (int lane = 0; lane < 32; ++lane) m = std::max(m, lane_window(lane, c0).count);
        for (int lane = 0; lane < 32; ++lane) {
          const int r = split ? lane % 16 : lane / g.lpr;
          const Window w = lane_window(lane, c0);
          for (int u = 0; u < m; ++u) {
            if (sizeof(R) == 8 && u >= w.count) continue;              // (not read)
            const int q = place<R>(w.first, w.count, u);
            if (q < 0 || q >= g.cap) return 2;                         // outside the warp's buffer
            if (u < w.count) {
              if (c0 + q >= pe) return 3;                              // not staged
              if (c0 + q < bound(r) || c0 + q >= bound(r + 1)) return 4;  // another row's
              if (split || lane % g.lpr == 0) {
                if (seen[c0 + q - p0]++) return 5;                     // read twice
                ++next[r];
              }
            }
          }
        }
        c0 += g.cap;
        if (c0 >= pe) break;
      }
      for (int r = 0; r < g.rpw; ++r)
        if (next[r] != bound(r + 1)) return 6;
    }
  return 0;
}

int main(int argc, char **argv) {
  std::vector<int> rp(1, 0);
  for (int v; std::scanf("%d", &v) == 1;) rp.push_back(rp.back() + v);
  for (int i = 1; i < argc; ++i) {
    const int nsp = std::atoi(argv[i]), f = walk<float>(rp, nsp), d = walk<double>(rp, nsp);
    if (f || d) {
      std::printf("%d columns: float %d, double %d\n", nsp, f, d);
      return 1;
    }
  }
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("window")
    src = d / "window.cu"
    src.write_text(PROGRAM)
    subprocess.run([nvcc, "-std=c++17", "-O1", "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a",
                    f"-I{CSRC}", f"-I{CSRC.parent.parent / 'include'}", str(src), "-o", str(d / "window")], check=True)
    return d / "window"


def _rows(kind):
    rng = np.random.default_rng(5)
    n = 1237
    r = rng.integers(8, 16, n)
    if kind == "uniform30":
        r[:] = 30
    elif kind == "hubs":
        r[[0, 7, 130, 131, 600, n - 1]] = [90, 150, 400, 60, 75, 333]
    elif kind == "empty":
        r[rng.random(n) < 0.5] = 0
    elif kind == "one":
        r[:] = 0
        r[5] = 1000
    return r


@pytest.mark.parametrize("kind", ["lattice", "uniform30", "hubs", "empty", "one"])
def test_every_read_stays_in_the_buffer(program, kind):
    cols = [str(c) for c in (2, 4, 8, 12, 16, 20, 24, 32, 36, 48, 64, 100, 128)]
    p = subprocess.run([program, *cols], input=" ".join(map(str, _rows(kind))), text=True, capture_output=True)
    assert p.returncode == 0, p.stdout
