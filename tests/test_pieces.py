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
    for f in (L.pc_doubles, L.pc_share):
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


def shares(pc, nx, nblocks):
    """(rhs, con) of the least and of the best shares of a context's scratch."""
    nn = [n + 9 for n in nx]
    plane, npts = (nx[0] + 1) * (nx[1] + 1), (nx[0] + 1) * (nx[1] + 1) * (nx[2] + 1)
    # the diagnostics and the adjoint: 33 values per vertex, 28 per interior one
    parts = 33 * nn[0] * nn[1] * nn[2] + 28 * npts
    least, best = (LL * 2)(), (LL * 2)()
    pc.pc_shares(LL(parts), LL(pc.pc_doubles(LL(npts), COMPONENTS)), LL(npts), LL(plane), CON,
                 nblocks, least, best)
    return parts, tuple(least), tuple(best)


def test_groups_of_an_odd_number_of_blocks(pc):
    """Three blocks of 112^3 whose scratch holds 1.5 of them: one block at a
    time."""
    nx = (112, 112, 112)
    _, _, (share, _) = shares(pc, nx, 3)
    assert share < pc.pc_doubles(LL(113 ** 3), COMPONENTS)
    rows = check(pc, nx, 0, 3, COMPONENTS, share)
    assert [r[:4] for r in rows] == [(b, 1, 0, 113) for b in range(3)]


@pytest.mark.parametrize("nx", [(8, 8, 8), (8, 8, 200), (200, 200, 8), (16, 16, 16),
                                (24, 24, 24), (33, 8, 12), (48, 48, 48), (160, 160, 160),
                                (300, 300, 300)])
def test_context_shares(pc, nx):
    """A context's shares hold the three arrays of the diagnostics and the
    adjoint, and planes enough for both passes on one block; the best ones are
    bounded."""
    for nblocks in (1, 3, 128, 512, 3424, 20000):
        parts, least, best = shares(pc, nx, nblocks)
        assert parts <= least[0] <= parts + 31
        assert least[0] <= best[0] and least[1] <= best[1]
        assert best[0] <= max(least[0] + least[0] // 16, 2 ** 29 // nblocks)
        assert best[1] == pc.pc_doubles(LL((nx[0] + 1) * (nx[1] + 1) * (nx[2] + 1)), CON)
        for s in (least, best):
            assert s[0] % 32 == 0 and s[1] % 32 == 0
            for comps, share in ((COMPONENTS, s[0]), (CON, s[1])):
                check(pc, nx, nblocks - 1, 1, comps, share)
                check(pc, nx, 0, min(nblocks, 5), comps, share)


def test_scratch_falls_back_when_the_device_is_full(pc):
    """A device that does not hold the best scratch gets the least one; one that
    does not hold that either refuses."""
    for nx, nblocks in (((128, 128, 128), 1), ((32, 32, 32), 64), ((16, 16, 16), 512)):
        _, least, best = shares(pc, nx, nblocks)
        for room, expect in ((sum(best) * nblocks, best), (sum(best) * nblocks - 1, least),
                             (sum(least) * nblocks, least), (sum(least) * nblocks - 1, None)):
            got, n = (LL * 2)(), LL()
            ok = pc.pc_reserve((LL * 2)(*least), (LL * 2)(*best), nblocks, LL(room), got,
                               C.byref(n))
            assert bool(ok) == (expect is not None)
            assert n.value == (sum(expect) * nblocks if expect else 0)
            if expect:
                assert tuple(got) == expect
