"""A context's memory does not grow with the number of calls: what a change of the
supports or a wider block of load cases replaces is given back, and the solves in
the new buffers end with the residual they report and repeat to the bit."""

import pytest
import torch

pytestmark = pytest.mark.gpu

NEL, LEVELS = (24, 12, 6), 2


def _ctx():
    from topogpu_b200.context import TopoContext

    return TopoContext(NEL, n_levels=LEVELS, mode="fp64")


def _masks():
    """Two supports with different numbers of free DoFs on the coarsest level (and another band)."""
    nx, ny, nz = NEL
    a = torch.ones(nx + 1, ny + 1, nz + 1, 3, dtype=torch.uint8)
    b = a.clone()
    a[0] = 0  # the face x = 0
    b[:, 0] = 0  # the face y = 0
    return a.reshape(-1).cuda(), b.reshape(-1).cuda()


TOL = 1e-9


def _solve(ctx, mask, E, B):
    ctx.set_problem(mask, B[0].contiguous())
    ctx.gmg_setup(E)
    X = torch.zeros_like(B)
    it, _, ok = ctx.block_pcg(B, X, tol=TOL, maxiter=300)
    assert ok
    x = torch.zeros_like(B[0])
    it1, _, ok = ctx.pcg(B[0].contiguous(), x, tol=TOL, maxiter=300)
    assert ok
    # the recursive residual is below TOL |b|; the true one leaves it by rounding only
    for u, b in [(x, B[0])] + list(zip(X, B)):
        b = b * mask
        assert float((b - ctx.matvec(u.contiguous(), E)).norm()) <= 2 * TOL * float(b.norm())
    return X, it, x, it1


def test_supports_alternate():
    g = torch.Generator().manual_seed(3)
    ctx = _ctx()
    E = (0.1 + torch.rand(ctx.n_elem, generator=g, dtype=torch.float64)).cuda()
    B = torch.randn(8, ctx.ndof, generator=g, dtype=torch.float64).cuda()
    want = [_solve(ctx, m, E, B) for m in _masks()]
    size = []
    for _ in range(3):
        for m, w in zip(_masks(), want):
            got = _solve(ctx, m, E, B)
            size.append(ctx.workspace_bytes())
            assert got[1] == w[1] and torch.equal(got[0], w[0])
            assert got[3] == w[3] and torch.equal(got[2], w[2])
    assert size[0:2] == size[2:4] == size[4:6]
    ctx.close()


def test_block_widths_change():
    g = torch.Generator().manual_seed(4)
    ctx = _ctx()
    m = _masks()[0]
    E = (0.1 + torch.rand(ctx.n_elem, generator=g, dtype=torch.float64)).cuda()
    B = torch.randn(8, ctx.ndof, generator=g, dtype=torch.float64).cuda()
    first = {}
    for nv in (2, 5, 8):
        first[nv] = _solve(ctx, m, E, B[:nv].contiguous())[0]
    size = ctx.workspace_bytes()
    for nv in (2, 8, 5, 2):
        assert torch.equal(_solve(ctx, m, E, B[:nv].contiguous())[0], first[nv])
        assert ctx.workspace_bytes() == size
    other = _ctx()
    _solve(other, m, E, B)
    assert other.workspace_bytes() == size  # the narrower workspaces are gone
    other.close()
    ctx.close()
