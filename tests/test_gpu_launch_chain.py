"""Overlapped kernel launches inside V-cycles and PCG iterations: a kernel
that read what the one before was still writing would change the bits from
call to call, or against a solve that runs the same V-cycle column by column.
Sizes: levels of one CTA, one wave and several waves, rows that end inside a
128-byte line, direct launches and graph replays, one and several columns."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _problem(nel, precision, **kw):
    from topogpu_b200.state import StateSolver

    nx, ny, nz = nel
    nn = (nx + 1) * (ny + 1) * (nz + 1)
    free = torch.ones(nn, 3, dtype=torch.uint8)
    free[: (ny + 1) * (nz + 1)] = 0  # the face x = 0
    F = torch.zeros(nn, 3, dtype=torch.float64)
    F[-1, 2] = -1.0
    s = StateSolver(nel, free.reshape(-1).numpy(), F.reshape(-1).numpy(), precision=precision, **kw)
    g = torch.Generator().manual_seed(7)
    rho = (0.3 + 0.7 * torch.rand(nx * ny * nz, generator=g, dtype=torch.float64)).cuda()
    return s, rho, g


@pytest.mark.parametrize("precision", ["fp64", "fp32", "mixed"])
@pytest.mark.parametrize("nel,levels", [((8, 4, 4), 2), ((24, 12, 6), 2), ((61, 30, 23), 3), ((96, 48, 48), 4)])
def test_vcycle_bits_repeat(nel, levels, precision):
    s, rho, g = _problem(nel, precision, n_levels=levels)
    s.ctx.gmg_setup(s.ctx.modulus(rho, 3.0, 1.0, 1e-9))
    r = (torch.randn(s.ctx.ndof, generator=g, dtype=torch.float64).cuda() * s.free_mask).to(s.ctx.vec_dtype)
    torch.cuda.synchronize()
    z0 = s.ctx.gmg_apply(r).clone()
    torch.cuda.synchronize()
    for i in range(50):
        z = s.ctx.gmg_apply(r)
        if i % 2:
            torch.cuda.synchronize()
        assert torch.equal(z, z0), i
    s.close()


@pytest.mark.parametrize("nel,levels", [((24, 12, 6), 2), ((48, 24, 24), 4)])
def test_solve_bits_repeat(nel, levels):
    s, rho, _ = _problem(nel, "fp64", n_levels=levels, warm_start=False)
    c0, dc0 = s.solve(rho)
    u0 = s.displacement().clone()
    for _ in range(5):
        c, dc = s.solve(rho)
        assert c == c0 and torch.equal(dc, dc0) and torch.equal(s.displacement(), u0)
    s.close()


@pytest.mark.parametrize("nel,levels,nv", [((17, 9, 5), 2, 3), ((96, 48, 48), 4, 8)])
def test_block_solve(nel, levels, nv):
    """The block solve against one solve per column: both end with a residual of
    at most tol |b|, so in the K^-1 inner product they lie 2 tol |b| apart; the
    compliances F.u differ by at most 2 tol |b| |u| (u = K^-1 b)."""
    tol = 1e-10
    s, rho, g = _problem(nel, "fp64", n_levels=levels, tol=tol, warm_start=False)
    B = torch.randn(nv, s.ctx.ndof, generator=g, dtype=torch.float64).cuda() * s.free_mask
    c0, U0 = s.solve_block(rho, B)
    assert s.last_converged
    for _ in range(3):
        c, U = s.solve_block(rho, B)
        assert c == c0 and torch.equal(U, U0)
    for j in range(nv):
        u = torch.zeros(s.ctx.ndof, dtype=torch.float64, device="cuda")
        _, _, ok = s.ctx.pcg(B[j].contiguous(), u, tol, 800)
        assert ok
        assert abs(float(torch.dot(B[j], u)) - c0[j]) <= 2 * tol * float(B[j].norm() * u.norm())
    s.close()
