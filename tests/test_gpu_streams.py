"""One context used with two streams: operators on different blocks whose
registers do not overlap need no ordering between their streams."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
PUNC = dict(diss=0.02, chi_div_floor=1e-5, damp_kappa1=0.02, shift_eta=2.0, r_max_con=1e300)


def make(nb, nx, contract):
    import z4c_b200 as Z
    from z4c_b200 import initial_data as ID
    h = 0.25
    lim = [0.5 * b * n * h for b, n in zip(nb, nx)]
    mesh = Z.Mesh(nb, nx, [-v for v in lim], lim, "outflow")
    ctx = Z.Z4c(mesh, Z.default_params(**PUNC), "rk4")
    ctx.set_contract(contract)
    ID.load_adm(ctx, ID.punctures(mesh, ctx.params, masses=(0.5,), centres=((0.53, 0.11, 0.07),),
                                  shift=(0.2, -0.1, 0.05)))
    ctx.evolve(0.25 * h, 1)
    ctx.sync()
    return Z, ctx


@pytest.mark.parametrize("contract", [False, True])
@pytest.mark.parametrize("nx", [(16, 16, 16), (40, 24, 22)])
def test_blocks_on_alternating_streams(nx, contract):
    """Right-hand sides of four blocks, and psi4 of a fifth, enqueued on two
    streams in turn without a wait between them: the bits of the same calls on
    one stream."""
    import torch
    Z, ctx = make((5, 1, 1), nx, contract)

    def run(streams):
        for reg in (Z.REG_RHS, Z.REG_WEYL):
            ctx.upload(reg, np.zeros(ctx.shape(reg)))
        torch.cuda.synchronize()
        for _ in range(12):
            for b in range(4):
                ctx.set_stream(streams[b % len(streams)].cuda_stream)
                ctx.Z4cRHS(Z.REG_U, Z.REG_RHS, b)
            ctx.set_stream(streams[-1].cuda_stream)
            ctx.Z4cWeyl(block=4)
        torch.cuda.synchronize()
        return ctx.download(Z.REG_RHS), ctx.download(Z.REG_WEYL)

    streams = [torch.cuda.Stream() for _ in range(2)]
    alone = run(streams[:1])
    both = run(streams)
    ctx.close()
    for a, b in zip(alone, both):
        assert np.array_equal(a, b, equal_nan=True)  # psi4 is NaN outside the interior


@pytest.mark.parametrize("contract", [False, True])
@pytest.mark.parametrize("nx", [(16, 16, 16), (40, 24, 22)])
def test_constraints_beside_right_hand_sides(nx, contract):
    """Constraints of single blocks and of the mesh on one stream, right-hand
    sides of the mesh on another: the bits of the same calls on one stream."""
    import torch
    Z, ctx = make((3, 1, 1), nx, contract)
    ctx.Z4cToADM()

    def run(streams):
        for reg in (Z.REG_RHS, Z.REG_CON):
            ctx.upload(reg, np.zeros(ctx.shape(reg)))
        torch.cuda.synchronize()
        for _ in range(12):
            ctx.set_stream(streams[0].cuda_stream)
            ctx.Z4cRHS()
            ctx.set_stream(streams[-1].cuda_stream)
            for b in (0, 1, 2, -1):
                ctx.ADMConstraints(block=b)
        torch.cuda.synchronize()
        return ctx.download(Z.REG_RHS), ctx.download(Z.REG_CON)

    streams = [torch.cuda.Stream() for _ in range(2)]
    alone = run(streams[:1])
    both = run(streams)
    ctx.close()
    for a, b in zip(alone, both):
        assert np.array_equal(a, b)
