"""The candidate rounds of the pair kernels' neighbour searches (csrc/mf_search.h): no lane of a warp
may load a candidate record past the array's padding, whatever the lengths of the columns that its
warp's other lanes go through. The kernels' loops replayed on the host for whole systems: the FP64
and mixed searches (a column at a time, the warp's lanes together) and the differentiable step's
(each lane through its own columns)."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent

REPLAY = r"""
#include <algorithm>
#include "mf_search.h"
using namespace mf;

// particle q's column c of the window: its particles' range in the sorted order
static void column(const int *off, int nx, int ny, const int *cell, int q, int c, bool act, int &j0, int &j1) {
  const int gi = cell[q] / ny, gj = cell[q] % ny, ii = gi - 2 + c;
  const bool in = act && c >= 0 && c < 5 && ii >= 0 && ii < nx;
  j0 = in ? off[ii * ny + std::max(gj - 2, 0)] : 0;
  j1 = in ? off[ii * ny + std::min(gj + 3, ny)] : 0;
}

// the largest index loaded (-1: a lane went below 0) by a system's warps at G lanes per particle;
// own: each lane goes through its own columns
extern "C" int largest_index(const int *off, int nx, int ny, const int *cell, int N, int G, int own) {
  const int per = 32 / G, U = CAND_STEP / G;
  int top = 0;
  auto load = [&](int jb, int sub) {
    for (int u = 0; u < U; ++u) {
      const int j = jb + u * G + sub;
      if (j < 0) top = -1;
      if (top >= 0) top = std::max(top, j);
    }
  };
  for (int q0 = 0; q0 < N; q0 += per) {
    int jb[32], j1[32], col[32];
    auto any = [&](auto f) {
      for (int l = 0; l < 32; ++l)
        if (f(l)) return true;
      return false;
    };
    auto q_of = [&](int l) { return q0 + l / G; };
    if (!own) {
      for (int c = 0; c < 5; ++c) {
        for (int l = 0; l < 32; ++l) column(off, nx, ny, cell, std::min(q_of(l), N - 1), c, q_of(l) < N, jb[l], j1[l]);
        while (any([&](int l) { return jb[l] < j1[l]; }))
          for (int l = 0; l < 32; ++l) {
            load(jb[l], l % G);
            jb[l] = next_round(jb[l], N);
          }
      }
    } else {
      for (int l = 0; l < 32; ++l) jb[l] = j1[l] = 0, col[l] = -1;
      do {
        for (int l = 0; l < 32; ++l) {
          while (jb[l] >= j1[l] && col[l] < 5)
            column(off, nx, ny, cell, std::min(q_of(l), N - 1), ++col[l], q_of(l) < N, jb[l], j1[l]);
          load(jb[l], l % G);
          jb[l] = next_round(jb[l], N);
        }
      } while (any([&](int l) { return col[l] < 5; }));
    }
  }
  return top;
}
extern "C" int padding() { return CAND_PAD; }
"""


@pytest.fixture(scope="module")
def replay(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("rounds")
    (d / "replay.cpp").write_text(REPLAY)
    r = subprocess.run([gxx, "-std=c++17", "-O2", "-shared", "-fPIC", "-I",
                        str(ROOT / "mfree_iwf-ul_cut_gpu_b200" / "csrc"), "-o", str(d / "replay.so"),
                        str(d / "replay.cpp")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return C.CDLL(str(d / "replay.so"))


def cells_of(kind, n, seed):
    """Cells (sorted) of n particles on a grid of about 2.25 particles a cell."""
    rng = np.random.default_rng(seed)
    side = max(1, int(round((n / 2.25) ** 0.5)))
    nx, ny = (side + 4, side + 4) if kind != "flat" else (max(5, n // 12), 7)
    cell = rng.integers(0, nx, n) * ny + rng.integers(0, ny, n)
    if kind == "lattice":
        x, y = np.divmod(np.arange(n), int(round(1.5 * side)) or 1)
        cell = (x / 1.5 + rng.uniform(0, 0.2, n)).astype(int) % nx * ny + (y / 1.5 + rng.uniform(0, 0.2, n)).astype(int)
    elif kind == "crowded":  # a crowded cell, and a few particles after it in the order
        few = min(3, n - 1)
        cell[: min(400, n - few)] = (nx - 2) * ny + ny // 2
        cell[n - few:] = (nx - 1) * ny + np.arange(ny // 2, ny // 2 + few) % ny
    return np.sort(np.minimum(cell, nx * ny - 1)).astype(np.int32), nx, ny


@pytest.mark.parametrize("kind", ["lattice", "flat", "random", "crowded"])
@pytest.mark.parametrize("n", [1, 9, 33, 1000, 7096, 31166])
def test_rounds_stay_in_the_padding(replay, kind, n):
    cell, nx, ny = cells_of(kind, n, n)
    off = np.concatenate([[0], np.cumsum(np.bincount(cell, minlength=nx * ny))]).astype(np.int32)
    ptr = lambda a: a.ctypes.data_as(C.c_void_p)
    for lanes in (1, 2, 4):
        for own in (0, 1):
            top = replay.largest_index(ptr(off), nx, ny, ptr(cell), n, lanes, own)
            assert 0 <= top < n + replay.padding(), (lanes, own, top)
