"""CPU: a CTA's place in a launch (csrc/indexing.h), compiled for the host: every tile once in all grids the rule leaves to that order, and
quotients that are exact where they are said to be; and the grids beyond it, which take other kernels."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import pytest

from aotriton_b200 import cabi
from test_host_fake_device import _bwd_args, fake      # noqa: F401 (a fixture)

CSRC = Path(__file__).resolve().parent.parent / "aotriton_b200" / "csrc"
PROGRAM = r"""
#include "indexing.h"
#include <cstdio>
#include <set>
#include <random>
#include <tuple>
using namespace ab200;
int bad = 0;
template <bool S> void every_tile_once(int nx, int nh, int nz) {
  std::set<std::tuple<int, int, int>> seen;
  for (int bz = 0; bz < nz; ++bz) for (int by = 0; by < nh; ++by) for (int bx = 0; bx < nx; ++bx) {
    int x, h, z;
    tile_of_block<S>(bx, by, bz, nx, nh, nz, x, h, z);
    if (x < 0 || x >= nx || h < 0 || h >= nh || z < 0 || z >= nz || !seen.insert({x, h, z}).second) ++bad;
  }
}
template <bool S> void in_range(int nx, int nh, int nz) {
  std::mt19937_64 g(1);
  std::set<std::tuple<int, int, int>> at, seen;
  for (int i = 0; i < 20000; ++i) {
    int bx = i < 4 ? (i & 1 ? nx - 1 : 0) : (int)(g() % nx), by = i < 4 ? (i & 2 ? nh - 1 : 0) : (int)(g() % nh), bz = i == 1 ? nz - 1 : (int)(g() % nz), x, h, z;
    tile_of_block<S>(bx, by, bz, nx, nh, nz, x, h, z);
    at.insert({bx, by, bz});
    if (x < 0 || x >= nx || h < 0 || h >= nh || z < 0 || z >= nz) ++bad; else seen.insert({x, h, z});
  }
  if (seen.size() != at.size()) ++bad;
}
int main() {
  if (beyond_tile_order(1 << 20, 32, 31) || !beyond_tile_order(1, 65535, 65535) || !beyond_tile_order(1 << 26, 1, 1)) ++bad;
  auto check = [](int a, int b) {
    bad += quick_div_any(a, b) != a / b;
    if (a < 1 << 24 || a / b < 1 << 22) bad += quick_div(a, b) != a / b;
  };
  for (int a : {0, 1, 2, 7, 147, 148, 149, (1 << 24) - 1, 1 << 24, (1 << 28) + 9, INT32_MAX - 1, INT32_MAX})
    for (int b : {1, 2, 3, 5, 7, 8, 24, 148, 65535, 1 << 24, INT32_MAX}) check(a, b);
  std::mt19937_64 g(2);
  for (int i = 0; i < 4000000; ++i) {
    const int a = (int)(g() & INT32_MAX) >> (g() % 31), b = ((int)(g() & INT32_MAX) >> (g() % 31)) | 1, c = 8 * (1 + (int)(g() % 64));
    check(a, b);
    check(a, c);
  }
  std::printf("%d ", bad); bad = 0;
  for (int nx : {1, 2, 5, 17}) for (int nh : {1, 3, 32, 40}) for (int nz : {1, 2, 7}) every_tile_once<true>(nx, nh, nz), every_tile_once<false>(nx, nh, nz);
  std::printf("%d ", bad); bad = 0;
  for (auto [nx, nh, nz] : {std::tuple{1, 65535, 32768}, {2, 65535, 16384}, {3, 65535, 10922}, {INT32_MAX / 32, 1, 1}, {INT32_MAX / 32, 2, 16}, {1 << 20, 2, 1023}})
    if (beyond_tile_order(nx, nh, nz)) ++bad; else in_range<true>(nx, nh, nz), in_range<false>(nx, nh, nz);
  std::printf("%d\n", bad);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a host compiler")
def test_places(tmp_path):
    src, exe = tmp_path / "places.cc", tmp_path / "places"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++20", "-fsanitize=signed-integer-overflow", "-fno-sanitize-recover", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split() == ["0", "0", "0"]


@pytest.mark.parametrize("B,H,S,launches", [
    (16383, 65535, 1, 2), (16384, 65535, 1, 2), (16385, 65535, 1, 3),      # the joint launch's 2 x 65535 x B CTAs
    (1, 1, 32 * ((1 << 25) - 1), 2), (1, 1, 32 << 25, 3)])                 # 32 heads of its row tiles
def test_grids_beyond_the_order_take_other_kernels(fake, B, H, S, launches):      # noqa: F811
    a = _bwd_args(dtype=cabi.DTYPE_FP32, D=4, B=B, Hq=H, Hk=H, S=S)
    for i, v in enumerate((a.q, a.out, a.dout, a.dq, a.k, a.v, a.dk, a.dv)):      # (apart, whatever their size)
        v.ptr = (i + 1) << 38
    a.lse, a.delta = 10 << 38, 11 << 38
    n0 = fake.ab200_launch_count()
    assert fake.ab200_attn_bwd(C.byref(a), None) == 0 and fake.ab200_last_bwd_family() == 1
    assert fake.ab200_launch_count() - n0 == launches      # preprocess, and dK/dV and dQ in one or two
