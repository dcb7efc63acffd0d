"""The derivative pass in pieces, where its scratch does not hold every block
(csrc/z4c_pieces.h): the same fields as one block of 160^3, whose planes run in
slabs, as eight blocks of 80^3, which run in two groups, and as single blocks of
80^3, whole; and the constraints of a context that found the device full.  A
vertex's right-hand side, stage output and constraints depend on its own
stencils only, so every decomposition gives the same values."""
import pytest

pytestmark = pytest.mark.gpu
N, NG, H = 80, 4, 0.25
PUNC = dict(diss=0.02, chi_div_floor=1e-5, damp_kappa1=0.02, shift_eta=2.0, r_max_con=1e300)


class Register:
    def __init__(self, ctx, reg):
        self.__cuda_array_interface__ = dict(shape=ctx.shape(reg), typestr="<f8", version=3,
                                             data=(ctx.device_ptr(reg), False))


def view(ctx, reg):
    import torch
    return torch.as_tensor(Register(ctx, reg), device="cuda")


def fields():
    """Smooth fields on the vertices of the 160^3 grid with its ghosts:
    [22][169][169][169], per cent waves around flat space, the shift of both
    signs."""
    import torch
    import z4c_b200 as Z
    n = 2 * N + 1 + 2 * NG
    x = torch.arange(n, dtype=torch.float64, device="cuda") * H
    g = torch.Generator().manual_seed(5)
    u = torch.zeros((22, n, n, n), dtype=torch.float64, device="cuda")
    for v in range(22):
        for _ in range(2):
            k = (torch.rand(3, generator=g, dtype=torch.float64) * 1.6 - 0.8).tolist()
            a, ph = (0.02 * (0.3 + torch.rand(1, generator=g)).item(),
                     6.0 * torch.rand(1, generator=g).item())
            u[v] += a * torch.sin(k[0] * x + k[1] * x[:, None] + k[2] * x[:, None, None] + ph)
    for v in (Z.CHI, Z.GXX, Z.GYY, Z.GZZ, Z.ALPHA):
        u[v] += 1.0
    return u


def block(full, at):
    """The block of 80^3 at position `at` (x, y, z) of the 2^3 blocks."""
    s = [slice(a * N, a * N + N + 1 + 2 * NG) for a in at]
    return full[:, s[2], s[1], s[0]]


def interior(f):
    return f[..., NG:-NG, NG:-NG, NG:-NG]


POSITIONS = [(i, j, k) for k in range(2) for j in range(2) for i in range(2)]  # block order


def outputs(nb, nx, u, contract, integ, full=False):
    """Registers after a right-hand side, a stage and the constraints of u
    [block][22][k][j][i], and the kernels launched by the first and the last."""
    import torch
    import z4c_b200 as Z
    mesh = Z.Mesh((nb,) * 3, (nx,) * 3, (0.0,) * 3, (nb * nx * H,) * 3, "outflow")
    taken = fill_device(nb ** 3, nx) if full else None
    ctx = Z.Z4c(mesh, Z.default_params(**PUNC), integ)
    del taken
    torch.cuda.empty_cache()
    ctx.set_contract(contract)
    view(ctx, Z.REG_U).copy_(u)
    if integ == "rk4":
        view(ctx, Z.REG_U1).copy_(u.flip(1))
    torch.cuda.synchronize()
    ctx.Z4cToADM()
    out, n0 = [], Z.kernel_launches()
    ctx.ADMConstraints()
    n1 = Z.kernel_launches()
    ctx.Z4cRHS()
    n2 = Z.kernel_launches()
    ctx.sync()
    out += [interior(view(ctx, r)).clone() for r in (Z.REG_CON, Z.REG_RHS)]
    if integ == "rk4":
        ctx.rhs_stage(2, 0.01)
        regs = (Z.REG_U1, Z.REG_W)
    else:
        ctx.stage(1, 0.01)
        regs = (Z.REG_K1, Z.REG_W)
    ctx.sync()
    out += [interior(view(ctx, r)).clone() for r in regs]
    torch.cuda.synchronize()
    ctx.close()
    return out, (n1 - n0, n2 - n1)


def fill_device(nblocks, nx):
    """Takes the device's memory but for what a low-storage context of nx^3 blocks
    needs beside its constraints' scratch, and half of that."""
    import torch
    nvol, npts = (nx + 9) ** 3, (nx + 1) ** 3
    # u, w, rhs, u1, adm, con, weyl and the inverse metric; derivatives, Ricci
    # and advection parts of the scratch, then half of the constraints' 63
    need = 8 * nblocks * ((4 * 22 + 17 + 7 + 2 + 6 + 33) * nvol + (28 + 63 // 2) * npts)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    return torch.empty(free - need - (64 << 20), dtype=torch.uint8, device="cuda")


def test_context_on_a_full_device_runs_in_smaller_pieces():
    """Where the preferred scratch is not to be had the context takes the least:
    the constraints plane by plane, with the same values."""
    import torch
    u = fields()
    best, n = outputs(1, 2 * N, u[None], False, "rk4")
    least, m = outputs(1, 2 * N, u[None], False, "rk4", full=True)
    assert n[0] == 2 and m[0] == 2 * (2 * N + 1)
    for a, b in zip(best, least):
        assert torch.equal(a, b)


@pytest.mark.parametrize("contract,integ", [(False, "rk4"), (True, "rk4"), (False, "bt_rk4")])
def test_pieces_give_the_whole_blocks_values(contract, integ):
    import torch
    u = fields()
    slabs, ns = outputs(1, 2 * N, u[None], contract, integ)
    groups, ng = outputs(2, N, torch.stack([block(u, p) for p in POSITIONS]), contract, integ)
    # right-hand side: two launches per piece, and Kreiss-Oliger on the exact path
    ko = 0 if contract else 1
    assert ns == (2, 2 * 3 + ko) and ng == (2, 2 * 2 + ko)
    for b, (i, j, k) in enumerate(POSITIONS):
        whole, nw = outputs(1, N, block(u, (i, j, k))[None], contract, integ)
        assert nw == (2, 2 + ko)
        for w, g, s in zip(whole, groups, slabs):
            sub = s[0, :, k * N:k * N + N + 1, j * N:j * N + N + 1, i * N:i * N + N + 1]
            assert torch.isfinite(w).all() and w.abs().max() > 0
            assert torch.equal(w[0], g[b])
            if contract:  # tiles of other widths may round their sums apart
                assert (w[0] - sub).abs().max() <= 1e-12 * w.abs().max()
            else:
                assert torch.equal(w[0], sub)
