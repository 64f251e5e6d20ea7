"""Load cases whose residuals are dependent, or become so: block PCG's Gram matrices
lose definiteness, and the columns that are left are solved one after another, each to
the tolerance asked for."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _context(nel, levels, mode, seed):
    from topogpu_b200.context import TopoContext

    ctx = TopoContext(nel, n_levels=levels, mode=mode)
    g = torch.Generator().manual_seed(seed)
    nx, ny, nz = nel
    mask = torch.ones(nx + 1, ny + 1, nz + 1, 3, dtype=torch.uint8)
    mask[0] = 0
    mask = mask.reshape(-1).cuda()
    E = (0.1 + torch.rand(ctx.n_elem, generator=g, dtype=torch.float64)).cuda()
    B = torch.randn(7, ctx.ndof, generator=g, dtype=torch.float64).cuda()
    return ctx, mask, E, B


def _solve(ctx, mask, E, B, tol):
    ctx.set_problem(mask, B[0].contiguous())
    ctx.gmg_setup(E)
    X = torch.zeros_like(B)
    it, rr, ok = ctx.block_pcg(B, X, tol=tol, maxiter=400)
    assert ok and 0 < it <= 400
    for u, b, r in zip(X, B * mask, rr):
        true = float((b - ctx.matvec(u.contiguous(), E)).norm())
        # the recursive residual is below tol |b|; the true one leaves it by rounding only
        assert true <= 2 * tol * float(b.norm()) and r <= tol
    return X


@pytest.mark.parametrize("mode, tol", [("fp64", 1e-9), ("fp32", 1e-5), ("mixed", 1e-5)])
def test_dependent_loads(mode, tol):
    ctx, mask, E, B = _context((24, 12, 6), 2, mode, 3)
    B[3] = B[1]
    B[5] = B[0] - 2.0 * B[2]
    X = _solve(ctx, mask, E, B, tol)
    # energy norm |x - K^-1 b| <= |r| / sqrt(lambda_min) for either column: compared through K
    d = ctx.matvec((X[3] - X[1]).contiguous(), E)
    assert float(d.norm()) <= 4 * tol * float((B[1] * mask).norm())
    ctx.close()


def test_residuals_that_become_dependent():
    # one level: many iterations with a BF16 smoother on 7 dense columns
    ctx, mask, E, B = _context((8, 6, 5), 1, "mixed", 6)
    _solve(ctx, mask, E, B, 1e-5)
    ctx.close()


def test_iteration_cap_is_kept():
    ctx, mask, E, B = _context((24, 12, 6), 2, "fp64", 4)
    B[1] = B[0]
    ctx.set_problem(mask, B[0].contiguous())
    ctx.gmg_setup(E)
    X = torch.zeros_like(B)
    it, rr, ok = ctx.block_pcg(B, X, tol=1e-12, maxiter=3)
    assert not ok and it <= 3 and max(rr) > 1e-12
    ctx.close()
