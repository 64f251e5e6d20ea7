"""The density filter takes every radius whose element has at most 1331 neighbours
within it (rmin up to 6.78), also where the radius exceeds the mesh."""

import numpy as np
import pytest
import torch

from oracle import design

pytestmark = pytest.mark.gpu

NELS = [(17, 13, 15), (40, 5, 6)]


def _ctx(nel):
    from topogpu_b200.context import TopoContext

    return TopoContext(nel, n_levels=1, mode="fp64")


@pytest.mark.parametrize("rmin", [0.7, 1.0, 5.999, 6.0, 6.4, 6.78])
@pytest.mark.parametrize("nel", NELS)
def test_filter_and_transpose(nel, rmin):
    H = design.filter_matrix(nel, rmin)
    x = np.random.default_rng(5).uniform(0.1, 1.0, H.shape[0])
    ctx = _ctx(nel)
    # positive terms: at most 1331 + 1331 additions, two products and a division of relative error 2^-53 each
    rtol = 2700 * 2.0 ** -53
    for tr, ref in ((False, H @ x), (True, H.T @ x)):
        y = ctx.filter(rmin, torch.tensor(x, device="cuda"), transpose=tr).cpu().numpy()
        np.testing.assert_allclose(y, ref, rtol=rtol, atol=0.0)
    ctx.close()


@pytest.mark.parametrize("rmin", [6.79, 7.0, 20.0])
def test_larger_radii_are_refused(rmin):
    nel = NELS[0]
    ctx = _ctx(nel)
    x = torch.ones(int(np.prod(nel)), dtype=torch.float64, device="cuda")
    with pytest.raises(RuntimeError, match="too large"):
        ctx.filter(rmin, x)
    assert float((ctx.filter(1.5, x) - 1).abs().max()) < 1e-14
    ctx.close()


def test_projected_update_beyond_radius_six():
    nel, rmin = NELS[0], 6.3
    rng = np.random.default_rng(6)
    n = int(np.prod(nel))
    rho, dc, dv = rng.uniform(0.2, 0.8, n), -rng.uniform(0.1, 1.0, n), rng.uniform(0.5, 1.5, n)
    H = design.filter_matrix(nel, rmin)
    ref, evals = design.oc_update_projected(rho, dc, dv, 0.4, 0.2, H, 4.0, 0.5)
    ctx = _ctx(nel)
    t = [torch.tensor(v, device="cuda") for v in (rho, dc, dv)]
    out, k = ctx.oc_projected(rmin, *t, 4.0, 0.5, 0.4, 0.2)
    assert k == evals
    # the bisection ends on multipliers 1e-9 apart; the update moves by rho s t d(lambda) / (2 lambda)
    np.testing.assert_allclose(out.cpu().numpy(), ref, rtol=0.0, atol=1e-8)
    ctx.close()
