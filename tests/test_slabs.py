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


LENGTHS = r"""
#include "ek_slabs.h"
#include <cstdio>
#include <cstdlib>
int main(int, char ** a)
{
  const int       N = atoi(a[1]);
  const long long limit = atoll(a[2]), cell = atoll(a[3]), fixed = atoll(a[4]);
  std::printf("%d\n", ekc::slab_cells(N, limit, [&](int n) { return fixed + cell * n; }));
}
"""


@pytest.fixture(scope="module")
def lengths(tmp_path_factory):
    return _compile(tmp_path_factory.mktemp("lengths"), LENGTHS)


@pytest.mark.parametrize("N,limit,cell,fixed", [(1, 10, 1, 0), (10, 100, 1, 0), (9, 4, 1, 0), (10, 4, 1, 0), (10, 8, 2, 1),
                                                (16, 10, 1, 0), (17, 16, 1, 0), (512, 1 << 30, 110 << 20, 200 << 20),
                                                (7, 3, 5, 0), (100_000, 1000, 7, 3), (2_000_000_000, 1 << 40, 100, 0)])
def test_slab_lengths(lengths, N, limit, cell, fixed):
    n = int(subprocess.run([lengths, str(N), str(limit), str(cell), str(fixed)], check=True, capture_output=True,
                           text=True).stdout)
    most = max(1, min(N, (limit - fixed) // cell))  # cells that fit
    assert 1 <= n <= most
    assert n == -(-N // -(-N // most))  # the fewest slabs, equal but for the rounding


PLACE = r"""
#include "ek_slabs.h"
#include <cstdio>
#include <cstdlib>
int main(int, char ** a)
{
  const int       n0 = atoi(a[1]);
  const long long cell = atoll(a[2]), fixed = atoll(a[3]), room = atoll(a[4]);
  const int       n = ekc::place_slab(n0, [&](int n) { return fixed + cell * n; }, [&](long long bytes) {
    std::printf("%lld ", bytes);
    return bytes <= room;
  });
  std::printf("-> %d\n", n);
}
"""


@pytest.fixture(scope="module")
def place(tmp_path_factory):
    return _compile(tmp_path_factory.mktemp("place"), PLACE)


@pytest.mark.parametrize("n,cell,fixed,room,asked,want", [
    (9, 10, 5, 100, [95], 9), (9, 10, 5, 94, [95, 55], 5), (9, 10, 5, 20, [95, 55, 35, 25, 15], 1),
    (9, 10, 5, 14, [95, 55, 35, 25, 15], 0), (1, 10, 5, 15, [15], 1), (1, 10, 5, 3, [15], 0), (0, 10, 5, 100, [], 0)])
def test_workspace_placement(place, n, cell, fixed, room, asked, want):
    out = subprocess.run([place, str(n), str(cell), str(fixed), str(room)], check=True, capture_output=True,
                         text=True).stdout.split("->")
    assert [int(x) for x in out[0].split()] == asked and int(out[1]) == want
