"""The projected OC update keeps its candidates in vectors the context has anyway: no
memory is made by a call, and the calls before and after it keep their bits."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp64", "fp32", "mixed"])
@pytest.mark.parametrize("nel, levels", [((43, 21, 17), 3), ((9, 5, 3), 1)])
def test_no_memory_and_no_trace(mode, nel, levels):
    from topogpu_b200.context import TopoContext

    ctx = TopoContext(nel, n_levels=levels, mode=mode)
    g = torch.Generator().manual_seed(8)
    n = ctx.n_elem
    nx, ny, nz = nel
    mask = torch.ones(nx + 1, ny + 1, nz + 1, 3, dtype=torch.uint8)
    mask[0] = 0
    mask = mask.reshape(-1).cuda()
    rho = (0.3 + 0.4 * torch.rand(n, generator=g, dtype=torch.float64)).cuda()
    dc = -(0.1 + torch.rand(n, generator=g, dtype=torch.float64)).cuda()
    dv = (0.5 + torch.rand(n, generator=g, dtype=torch.float64)).cuda()
    b = torch.randn(ctx.ndof, generator=g, dtype=torch.float64).cuda() * mask
    E = ctx.modulus(rho)
    ctx.set_problem(mask, b)
    ctx.gmg_setup(E)
    r = b.to(ctx.vec_dtype)

    def update():
        return ctx.oc_projected(2.0, rho, dc, dv, 8.0, 0.5, 0.4, 0.2)

    def solve():
        x = torch.zeros_like(b)
        it, rr, ok = ctx.pcg(b, x, tol=1e-5, maxiter=400)
        return x, it, ok

    z0, (x0, it0, _) = ctx.gmg_apply(r), solve()
    size = ctx.workspace_bytes()
    out0, ev0 = update()
    assert torch.equal(ctx.gmg_apply(r), z0)
    out, ev = update()
    assert ev == ev0 and torch.equal(out, out0)
    x, it, _ = solve()
    assert it == it0 and torch.equal(x, x0)
    ctx.gmg_setup(E * 2.0)  # a new spectral bound, on vectors that held candidates
    update()
    ctx.gmg_setup(E)
    assert torch.equal(ctx.gmg_apply(r), z0)
    assert ctx.workspace_bytes() == size
    ctx.close()
