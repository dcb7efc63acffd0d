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
CON = 63  # of the constraints
LL = C.c_longlong


@pytest.fixture(scope="module")
def pc(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("pc") / "pc.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-o", out, SRC], check=True)
    L = C.CDLL(out)
    for f in (L.pc_doubles, L.pc_share, L.pc_context_share, L.pc_con_share):
        f.restype = LL
    return L


def chunks(pc, nx, block0, nblk, comps, share):
    rows = np.zeros((nblk * (nx[2] + 1) + 1, 5), np.int64)
    n = pc.pc_chunks((C.c_int * 3)(*nx), block0, nblk, comps, LL(share),
                     rows.ctypes.data_as(C.POINTER(LL)), len(rows))
    assert 0 < n <= len(rows)
    return [tuple(int(v) for v in r) for r in rows[:n]]


def check(pc, nx, block0, nblk, comps, share):
    """The pieces cover blocks block0 .. block0 + nblk - 1 once and stay inside
    these blocks' shares of the scratch."""
    plane, nk = (nx[0] + 1) * (nx[1] + 1), nx[2] + 1
    seen = np.zeros((nblk, nk), int)
    rows = chunks(pc, nx, block0, nblk, comps, share)
    for b, nb, ks, n, at in rows:
        assert nb >= 1 and n >= 1
        need = nb * pc.pc_doubles(LL(plane * n), comps)
        where = (nx, block0, nblk, share, (b, nb, ks, n, at), need)
        assert at >= block0 * share and at + need <= (block0 + nblk) * share, where
        seen[b - block0:b - block0 + nb, ks:ks + n] += 1
    assert (seen == 1).all(), (nx, nblk, share)
    return rows


@pytest.mark.parametrize("nx", [(8, 8, 8), (16, 16, 16), (22, 13, 18), (112, 112, 112)])
def test_pieces_stay_inside_the_shares_and_cover_the_mesh(pc, nx):
    plane, nk = (nx[0] + 1) * (nx[1] + 1), nx[2] + 1
    per = pc.pc_doubles(LL(plane * nk), COMPONENTS)
    for total in (1, 2, 3, 5, 7, 64):
        # two planes of a block up to the whole mesh
        for cap in sorted({total * (2 * plane + 64) * COMPONENTS, per // 2, per - 1, per, per + 1,
                           int(1.6 * per), 2 * per, 3 * per - 1, total * per // 2,
                           int(0.52 * total * per), total * per - 1, total * per}):
            share = pc.pc_share(LL(cap), total)
            assert share % 32 == 0 and share * total <= cap
            if (share // COMPONENTS - 32) // plane < 1:
                continue  # less than a plane per block: no context makes it
            check(pc, nx, 0, total, COMPONENTS, share)
            for b in {0, total // 2, total - 1}:  # a call on one block, or on the last ones
                check(pc, nx, b, 1, COMPONENTS, share)
                check(pc, nx, b, total - b, COMPONENTS, share)


def parts(nx):  # 33 values per vertex and 28 per interior vertex
    nn = [n + 9 for n in nx]
    return 33 * nn[0] * nn[1] * nn[2] + 28 * (nx[0] + 1) * (nx[1] + 1) * (nx[2] + 1)


def test_groups_of_an_odd_number_of_blocks(pc):
    """Three blocks of 112^3 whose scratch holds 1.5 of them: one block at a
    time."""
    nx = (112, 112, 112)
    per = pc.pc_doubles(LL(113 ** 3), COMPONENTS)
    share = pc.pc_context_share(LL(parts(nx)), LL(per), 3)
    assert share < per
    rows = check(pc, nx, 0, 3, COMPONENTS, share)
    assert [r[:4] for r in rows] == [(b, 1, 0, 113) for b in range(3)]


def test_context_shares(pc):
    """A context's share holds the three arrays of the diagnostics and the
    adjoint, and planes enough for the derivative pass on one block."""
    for nx in [(8, 8, 8), (8, 8, 200), (200, 200, 8), (16, 16, 16), (24, 24, 24), (33, 8, 12),
               (48, 48, 48), (160, 160, 160), (300, 300, 300)]:
        plane, nk = (nx[0] + 1) * (nx[1] + 1), nx[2] + 1
        per = pc.pc_doubles(LL(plane * nk), COMPONENTS)
        for nblocks in (1, 3, 128, 3424):
            share = pc.pc_context_share(LL(parts(nx)), LL(per), nblocks)
            assert share >= parts(nx) and share % 32 == 0
            assert share <= max(parts(nx) + parts(nx) // 16, 2 ** 29 // nblocks) + 32
            check(pc, nx, nblocks - 1, 1, COMPONENTS, share)
            check(pc, nx, 0, min(nblocks, 3), COMPONENTS, share)


def test_constraint_shares(pc):
    """The constraints' scratch: whole blocks up to 1 GiB on the mesh, at least
    a plane of every block."""
    for nx in [(8, 8, 8), (200, 200, 8), (16, 16, 16), (24, 24, 24), (33, 8, 12), (160, 160, 160)]:
        plane, nk = (nx[0] + 1) * (nx[1] + 1), nx[2] + 1
        per = pc.pc_doubles(LL(plane * nk), CON)
        for nblocks in (1, 3, 128, 512, 3424, 20000):
            share = pc.pc_con_share(LL(plane * nk), LL(plane), CON, nblocks)
            assert share % 32 == 0 and share <= per
            assert share == per or share * nblocks <= 2 ** 27 or share <= CON * (plane + 64)
            check(pc, nx, nblocks - 1, 1, CON, share)
            check(pc, nx, 0, min(nblocks, 5), CON, share)
