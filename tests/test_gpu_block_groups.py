"""Block solves whose V-cycle takes fewer columns at once than there are load cases
(little free memory): each column's preconditioned residual is the same operator, so
every solve ends below its tolerance, in as many iterations as the whole block needs,
give or take the one that rounding may decide."""

import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-9, "fp32": 1e-5, "mixed": 1e-5}


@pytest.mark.parametrize("mode, nel, levels", [("fp64", (24, 12, 6), 2), ("fp32", (24, 12, 6), 2), ("mixed", (24, 12, 6), 2),
                                               ("fp64", (21, 13, 9), 3), ("fp32", (21, 13, 9), 3), ("mixed", (21, 13, 9), 3),
                                               ("fp64", (8, 6, 5), 1), ("fp32", (8, 6, 5), 1)])
def test_groups_of_columns(mode, nel, levels):
    from topogpu_b200.context import TopoContext

    tol = TOL[mode]
    ctx = TopoContext(nel, n_levels=levels, mode=mode)
    g = torch.Generator().manual_seed(6)
    nx, ny, nz = nel
    mask = torch.ones(nx + 1, ny + 1, nz + 1, 3, dtype=torch.uint8)
    mask[0] = 0
    mask = mask.reshape(-1).cuda()
    E = (0.1 + torch.rand(ctx.n_elem, generator=g, dtype=torch.float64)).cuda()
    B = torch.randn(7, ctx.ndof, generator=g, dtype=torch.float64).cuda()
    ctx.set_problem(mask, B[0].contiguous())
    ctx.gmg_setup(E)

    def solve():
        X = torch.zeros_like(B)
        it, _, ok = ctx.block_pcg(B, X, tol=tol, maxiter=300)
        assert ok
        for u, b in zip(X, B * mask):
            # the recursive residual is below tol |b|; the true one leaves it by rounding only
            assert float((b - ctx.matvec(u.contiguous(), E)).norm()) <= 2 * tol * float(b.norm())
        return it, ctx.workspace_bytes()

    it0, size0 = solve()
    for columns in (5, 3, 2, 1):
        assert ctx._lib.topo_debug_block_columns(ctx._h, columns) == 0
        it, size = solve()
        assert abs(it - it0) <= 1 and size < size0
    ctx.close()
