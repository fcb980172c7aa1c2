"""The shared-memory layout of the fixed-point nonlocal kernel (csrc/nonlocal_fx_layout.h), compiled
as plain C++: every region holds what the kernel puts into it, none reaches into the next, and the
size that launches ask for covers the last one (a size without an entry table's end marker once let
the kernel write past its shared memory for some counts)."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sparc_gb300",
                    "csrc")

PROGRAM = r"""
#include <cstdio>
#include <initializer_list>
#include "nonlocal_fx_layout.h"
using namespace sgpu::nlfx;
int main()
{
    long bad = 0, n = 0;
    for (int jp : {10, 18})
        for (int rows = 1; rows <= 128; rows++)
            for (int ent : {1, 2, 15, 16, 17, 31, 128, 226, 227, 408, 409})
                for (int items = 1; items <= 128; items++) {
                    const auto L = regions<std::size_t>(0, rows, ent, items, jp);
                    const unsigned bytes = shared_bytes(rows, ent, items, jp);
                    const std::size_t r = rows, e = ent, i = items;
                    // start, bytes used and alignment of each region, in the order of the layout
                    const std::size_t reg[][3] = {
                        {L.tile, 8 * 128 * 33, 16},       {L.al, r * 32 * 8, 8},
                        {L.chi, e * jp * 8, 16},     {L.lps, e, 1},
                        {L.rows, r * 16, 16},        {L.items, i * 16, 16},
                        {L.ent0, (i + 1) * 4, 4},    {L.wsplit, i * 9 * 4, 4},
                        {bytes, 0, 16}};
                    for (int k = 0; k < 9; k++) {
                        if (reg[k][0] % reg[k][2]) bad++;
                        if (k < 8 && reg[k][0] + reg[k][1] > reg[k + 1][0]) bad++;
                    }
                    // the largest ranges that are built: 128 rows, 32 KB of Chi digits, an item
                    // per row at most
                    if (e * jp * 8 <= 32 * 1024 && items <= rows && bytes > 227 * 1024) bad++;
                    n++;
                }
    std::printf("%ld of %ld\n", bad, n);
    return bad != 0;
}
"""


def test_regions_hold_their_tables(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    src, exe = tmp_path / "layout.cpp", tmp_path / "layout"
    src.write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-I", CSRC, str(src), "-o",
                    str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
