"""Shared-memory layouts (make_layout) at sizes near the 227 KB of a CTA, on
the CPU: tile sizes and parked rows of relative lightcurves that fit (where the
rows are not parked, the allocation-free entry point runs a fraction of the fit
slots), places that may share memory, and places that may not."""
from __future__ import annotations

import subprocess

import pytest

from conftest import ROOT

PROGRAM = """
#include <cstdint>
#include <cstddef>
#include <cstdio>
#include <cstdlib>
struct float2 { float x, y; };
struct float4 { float x, y, z, w; };
#include "ps_engine.h"
int main(int, char **v)
{
    int a[6];
    for (int k = 0; k < 6; k++) a[k] = std::atoi(v[k + 1]);
    const int C = (a[1] + 1) * (a[1] + 1);
    const psg::SlotLayout L = psg::make_layout(a[0], C + 8, C + 6, 8 * a[2] * a[2], C, a[3], a[4], a[5]);
    std::printf("%zu %zu %zu %zu %zu %zu %d\\n", L.bytes, L.col, L.col + sizeof(double) * psg::gj_doubles(C + 6) + sizeof(int) * psg::gj_ints(C + 6), L.W, L.dave,
                L.phase, L.phase_tiles);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("layout")
    (d / "layout.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", str(ROOT / "include"), "-I", str(ROOT / "periodsearch_gb300" / "csrc"),
                    str(d / "layout.cpp"), "-o", str(d / "layout")], check=True)
    return d / "layout"


# form, Laplace degree, facet rows, points of a tile, basis mode, parked rows
@pytest.mark.parametrize("case", [(0, 5, 8, 32, 0, 0), (0, 8, 5, 32, 0, 0), (0, 8, 11, 8, 0, 0), (0, 2, 4, 32, 0, 1000),
                                  (0, 4, 6, 32, 0, 300), (0, 6, 6, 32, 0, 100), (0, 7, 6, 32, 0, 20),
                                  (1, 9, 7, 16, 0, 0), (0, 6, 6, 32, 0, 60), (0, 3, 4, 32, 0, 0)])
def test_layout_fits(program, case):
    out = subprocess.run([str(program), *map(str, case)], check=True, capture_output=True, text=True).stdout
    size, col, col_end, w, tiles_end, phase, phase_tiles = map(int, out.split())
    assert size <= 227 * 1024
    assert w <= col and col_end <= tiles_end          # the solvers' workspace over the tiles'
    assert 1 <= phase_tiles <= 12 and (phase_tiles == 1 or phase >= tiles_end)
    if case in ((0, 3, 4, 32, 0, 0), (0, 6, 6, 32, 0, 60)):
        assert phase_tiles == 12
