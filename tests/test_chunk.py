"""The planes-per-CTA rule of the 3D kernels (euler_kokkos_gb300/csrc/ek_chunk.h),
compiled as plain C++ on the host."""

import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "ek_chunk.h"
#include <cstdio>
#include <cstdlib>
#include <initializer_list>
int main(int, char ** a)
{
  const ekc::ChunkModel m[6] = { ekc::kChunkHydro64, ekc::kChunkHydro32, ekc::kChunkTrace64, ekc::kChunkTrace32,
                                 ekc::kChunkUpdate64, ekc::kChunkUpdate32 };
  if (atoi(a[3]) < 0) // rows of the 2D marches: nx, ny, -sms
  {
    const int nx[2] = { atoi(a[1]), atoi(a[1]) }, ny[2] = { atoi(a[2]), atoi(a[2]) };
    for (int n = 1; n <= 2; ++n)
      for (auto & x : { ekc::kChunkRows64, ekc::kChunkRows32 })
        std::printf("%d ", ekc::choose_rows(nx, ny, n, -atoi(a[3]), x));
    return 0;
  }
  for (auto & x : m)
    std::printf("%d ", ekc::choose_chunk(atoll(a[1]), atoi(a[2]), atoi(a[3]), x));
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("chunk")
    (d / "c.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "euler_kokkos_gb300", "csrc"), str(d / "c.cpp"),
                    "-o", str(d / "c")], check=True)
    return str(d / "c")


@pytest.mark.parametrize("columns,planes,sms", [(1, 2, 152), (1, 3, 1), (4, 32, 152), (6, 99, 152), (16, 64, 152),
                                                (256, 256, 152), (1156, 2, 152), (1 << 22, 7, 152), (1, 100000, 1)])
def test_chunks_cover_the_planes(program, columns, planes, sms):
    for kc in map(int, subprocess.run([program, str(columns), str(planes), str(sms)], check=True, capture_output=True,
                                      text=True).stdout.split()):
        assert 1 <= kc <= min(planes, 64)
        chunks = -(-planes // kc)
        assert chunks <= 65535 and (chunks - 1) * kc < planes <= chunks * kc
        if columns * planes <= sms:  # every plane its own SM
            assert kc == 1
        if columns >= 1000 * sms:  # plenty of tiles: no repeated end planes
            assert kc == planes


@pytest.mark.parametrize("nx,ny", [(1, 1), (2, 2), (64, 64), (28, 10_000_000), (1, 4_000_000), (1022, 518), (30000, 20000)])
def test_runs_of_rows(program, nx, ny):
    for rows in map(int, subprocess.run([program, str(nx), str(ny), "-152"], check=True, capture_output=True,
                                        text=True).stdout.split()):
        assert 1 <= rows <= min(ny, 64) and -(-ny // (4 * rows)) <= 65535
        if nx * ny <= 64 * 64:  # few warps: one row each
            assert rows == 1
