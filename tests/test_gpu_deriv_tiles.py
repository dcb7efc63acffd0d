"""The derivative and pointwise passes at the edges of their tiles: rows of
one, just over one and two tile widths, several tiles of either instance on
either axis, the smallest blocks, heights around the tile's, several blocks;
against the CPU oracle block by block.  The contracted path's fixed instance for
a block of 128^3 against the exact path."""
import numpy as np
import pytest

import z4c_oracle as O
from z4c_testlib import rel_err

pytestmark = pytest.mark.gpu
PUNC = dict(diss=0.02, chi_div_floor=1e-5, damp_kappa1=0.02, shift_eta=2.0, r_max_con=1e300)


@pytest.mark.parametrize("contract", [False, True])
@pytest.mark.parametrize("nb,nx", [
    ((1, 1, 1), (8, 8, 8)),      # the smallest block
    ((2, 1, 2), (17, 16, 9)),    # 18 columns, 17 rows: one full tile of the narrow instance
    ((1, 2, 1), (18, 17, 8)),    # 19 columns: the wide instance, two rows of tiles of 9
    ((1, 1, 1), (33, 8, 12)),    # 34 columns, 9 rows: one full tile of the wide instance
    ((1, 1, 1), (34, 9, 16)),    # 35 columns: two narrow tiles, an odd number of rows
    ((1, 1, 1), (67, 8, 16)),    # 68 columns: two full tiles of the wide instance
    ((1, 1, 1), (60, 25, 8)),    # wide, 2 x 3 tiles, the last of both axes cut off
    ((1, 1, 2), (70, 11, 37)),   # four narrow tiles, six chunks of planes
])
def test_rhs_matches_oracle_at_tile_edges(nb, nx, contract):
    import z4c_b200 as Z
    from z4c_b200 import initial_data as ID
    h = 0.25
    lim = [0.5 * b * n * h for b, n in zip(nb, nx)]
    mesh = Z.Mesh(nb, nx, [-v for v in lim], lim, "outflow")
    ctx = Z.Z4c(mesh, Z.default_params(**PUNC), "rk4")
    ctx.set_contract(contract)
    ID.load_adm(ctx, ID.punctures(mesh, ctx.params, masses=(0.5, 0.4),
                                  centres=((0.53, 0.11, 0.07), (-0.61, -0.2, 0.03)),
                                  shift=(0.2, -0.1, 0.05)))
    ctx.evolve(0.25 * h, 1)  # K, Theta and Gamma away from zero
    u = ctx.download(Z.REG_U)
    ctx.Z4cRHS()
    rhs = ctx.download(Z.REG_RHS)
    ctx.close()
    p = O.default_params(**PUNC)
    inner = (slice(None),) + (slice(4, -4),) * 3
    for b in range(mesh.nblocks):
        xs, dxs = mesh.block_coords(b)
        ref = O.rhs(O.Block(mesh.nx, dxs, xs), p, u[b])
        # the exact path agrees to the ulps of pow and cbrt, the contracted one
        # to rounding of sums whose terms are at most 1e3 times the result
        assert rel_err(rhs[b][inner], ref[inner]) <= 1e-12, b


def test_fixed_instance_of_128_cubed_matches_the_exact_path():
    """One block of 128^3: the contracted path evaluates its stencils in place.
    The exact path, which the oracle checks at other sizes, bounds it as the
    oracle bounds the contracted path there."""
    import z4c_b200 as Z
    from z4c_b200 import initial_data as ID
    mesh = Z.Mesh((1, 1, 1), (128, 128, 128), (-16.0,) * 3, (16.0,) * 3, "outflow")
    ctx = Z.Z4c(mesh, Z.default_params(**PUNC), "rk4")
    ID.load_adm(ctx, ID.punctures(mesh, ctx.params, masses=(0.5, 0.4),
                                  centres=((0.53, 0.11, 0.07), (-0.61, -0.2, 0.03)),
                                  shift=(0.2, -0.1, 0.05)))
    dt = 0.0625
    ctx.evolve(dt, 1)
    out = []
    for contract in (False, True):
        ctx.set_contract(contract)
        ctx.upload(Z.REG_U1, ctx.download(Z.REG_U)[:, ::-1].copy())
        ctx.Z4cRHS()
        rhs = ctx.download(Z.REG_RHS)
        ctx.rhs_stage(2, dt)
        out.append((rhs, ctx.download(Z.REG_W), ctx.download(Z.REG_U1)))
    ctx.close()
    inner = (slice(None), slice(None)) + (slice(4, -4),) * 3
    exact, contracted = out
    assert not np.array_equal(exact[0][inner], contracted[0][inner])
    for a, b in zip(contracted, exact):
        assert rel_err(a[inner], b[inner]) <= 1e-12
