"""The derivative and pointwise passes at the edges of their tiles: rows of
one, just over one and two tile widths, the smallest blocks, heights around
the tile's, several blocks; against the CPU oracle block by block."""
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
    ((1, 1, 2), (70, 11, 37)),   # three tiles, two chunks of planes
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
