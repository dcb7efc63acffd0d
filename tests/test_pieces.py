"""The pieces in which the derivative and pointwise passes run where their
scratch does not hold every block (csrc/z4c_pieces.h), on the CPU: every piece
fits the scratch, and together they cover every block and interior plane once.

tests/pieces/pieces_check.cpp wraps the header in a small C library built here
with g++."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from z4c_testlib import ROOT

SRC = os.path.join(ROOT, "tests", "pieces", "pieces_check.cpp")
COMPONENTS = 136  # of the right-hand side, per interior vertex


@pytest.fixture(scope="module")
def pc(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("pc") / "pc.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-o", out, SRC], check=True)
    L = C.CDLL(out)
    L.pc_doubles.restype = C.c_longlong
    return L


def chunks(pc, nx, nblk, comps, cap):
    rows = np.zeros((nblk * (nx[2] + 1) + 1, 4), np.intc)
    n = pc.pc_chunks((C.c_int * 3)(*nx), nblk, comps, C.c_longlong(cap),
                     rows.ctypes.data_as(C.POINTER(C.c_int)), len(rows))
    assert 0 < n <= len(rows)
    return [tuple(int(v) for v in r) for r in rows[:n]]


def check(pc, nx, nblk, comps, cap):
    plane, nk = (nx[0] + 1) * (nx[1] + 1), nx[2] + 1
    seen = np.zeros((nblk, nk), int)
    rows = chunks(pc, nx, nblk, comps, cap)
    for b, nb, ks, n in rows:
        assert nb >= 1 and n >= 1
        need = nb * pc.pc_doubles(C.c_longlong(plane * n), comps)
        assert need <= cap, (nx, nblk, cap, (b, nb, ks, n), need)
        seen[b:b + nb, ks:ks + n] += 1
    assert (seen == 1).all(), (nx, nblk, cap)
    return rows


@pytest.mark.parametrize("nx", [(8, 8, 8), (16, 16, 16), (22, 13, 18), (112, 112, 112)])
def test_pieces_fit_the_scratch_and_cover_the_mesh(pc, nx):
    plane, nk = (nx[0] + 1) * (nx[1] + 1), nx[2] + 1
    per = pc.pc_doubles(C.c_longlong(plane * nk), COMPONENTS)
    for nblk in (1, 2, 3, 5, 7, 64):
        # two planes of a block up to the whole mesh
        for cap in sorted({pc.pc_doubles(C.c_longlong(2 * plane), COMPONENTS) + 32 * COMPONENTS,
                           per // 2, per - 1, per, per + 1, int(1.6 * per), 2 * per, 3 * per - 1,
                           nblk * per // 2, int(0.52 * nblk * per), nblk * per - 1, nblk * per}):
            check(pc, nx, nblk, COMPONENTS, cap)


def test_groups_of_an_odd_number_of_blocks(pc):
    """Three blocks of 112^3 whose scratch (33 values per vertex and 28 per
    interior vertex) holds 1.5 of them: one block at a time."""
    nx = (112, 112, 112)
    cap = 3 * (33 * 121 ** 3 + 28 * 113 ** 3)
    rows = check(pc, nx, 3, COMPONENTS, cap)
    assert rows == [(b, 1, 0, 113) for b in range(3)]
