"""The slabs of the FP64 steps in passes (euler_kokkos_gb300/csrc/ek_slabs.h),
compiled as plain C++ on the host."""

import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

OFFSETS = r"""
#include "ek_slabs.h"
#include <cstdio>
#include <cstdlib>
template <int DIM>
static int check(int nx, int ny, int n)
{
  ekc::MhdSlab<DIM> S{};
  S.nx = nx, S.ny = DIM == 2 ? n : ny, S.nz = DIM == 2 ? 1 : n;
  const int ny_ = S.ny, nz_ = DIM == 2 ? 1 : n;
  int       bad = 0;
  const auto st = S.trace_stride();
  const __int128 cells = (__int128)(nx + 2) * (ny_ + 2) * (DIM == 3 ? n + 2 : 1);
  bad += (__int128)st != cells;
  // the first and last trace cell that the faces and edges read, every field
  const long long lo = S.tcell(-1, -1, DIM == 3 ? -1 : 0), hi = S.tcell(nx, ny_, DIM == 3 ? nz_ : 0);
  bad += lo != 0 || (__int128)hi != cells - 1;
  for (int f = 0; f < S.NT; ++f)
    bad += (__int128)ekc::field_offset(f, st) != (__int128)f * cells;
  bad += (__int128)hi + ekc::field_offset(S.NT - 1, st) != S.NT * cells - 1;
  bad += (__int128)S.slab_bytes() < (__int128)8 * S.NT * cells;
  // a tile's planes in shared memory stay 32 bits
  bad += sizeof(ekc::field_offset(3, 180)) != 4 || ekc::field_offset(46, 340) != 46 * 340;
  return bad;
}
int main(int, char ** a)
{
  const int nx = atoi(a[2]), ny = atoi(a[3]), n = atoi(a[4]);
  std::printf("%d\n", atoi(a[1]) == 2 ? check<2>(nx, ny, n) : check<3>(nx, ny, n));
}
"""


def _compile(d, source):
    (d / "c.cpp").write_text(source)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "euler_kokkos_gb300", "csrc"), str(d / "c.cpp"),
                    "-o", str(d / "c")], check=True)
    return str(d / "c")


@pytest.fixture(scope="module")
def offsets(tmp_path_factory):
    return _compile(tmp_path_factory.mktemp("offsets"), OFFSETS)


# 3942 x 3942: the last square plane whose fields stay below 2^31
@pytest.mark.parametrize("dim,nx,ny,n", [(3, 16, 8, 5), (3, 3942, 3942, 1), (3, 3943, 3943, 1), (3, 4000, 4000, 1),
                                         (3, 12000, 9000, 1), (2, 200, 136, 136), (2, 30_000_000, 3, 1)])
def test_trace_offsets_of_large_planes(offsets, dim, nx, ny, n):
    assert subprocess.run([offsets, str(dim), str(nx), str(ny), str(n)], check=True, capture_output=True,
                          text=True).stdout.strip() == "0"
