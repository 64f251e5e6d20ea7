"""The bracketing search of the filtered OC and the tap loop of the filter at
the places where they can go wrong.

The search evaluates other multipliers than run_simp's bisection but has to
return the sequential bisection's evaluation count and design: checked bit for
bit against a sequential restatement (pub_simp_solver.py:319-340) over
multipliers from far below to far above one, volume fractions that cannot be
reached from either side (the bisection then runs to an end of its bracket),
saturated and zero sensitivities, and column sums of both signs (the volume is
not monotone there, every midpoint is evaluated). The filter: extents below
and at the radius, so that rows are cut on both sides, against a dense
row-normalised matrix (a few ulps of a sum of positive terms: 1e-14)."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def sequential(rho, dc, dv, colsum, volfrac, move, rho_min=1e-3):
    l1, l2, k, rn = 0.0, 1e9, 0, rho
    while True:
        lm = 0.5 * (l1 + l2)
        rn = rho * np.sqrt(-np.minimum(dc, -1e-12) / (lm * np.maximum(dv, 1e-12)))
        rn = np.clip(np.clip(rn, rho - move, rho + move), rho_min, 1.0)
        k += 1
        if float(np.dot(rn, colsum)) / len(rho) > volfrac:
            l1 = lm
        else:
            l2 = lm
        if l2 - l1 < 1e-9 or k >= 100:
            return rn, k


def _case(name, n, rng):
    rho = rng.uniform(0.01, 1.0, n)
    dc = -rng.gamma(1.0, 1.0, n)
    dv = rng.uniform(0.8, 1.0, n)
    col, vf = dv.copy(), 0.3
    if name == "small":
        dc = dc * 1e-6
    elif name == "large":
        dc = dc * 1e4
    elif name == "decades":
        dc = dc * 10.0 ** rng.uniform(-8, 2, n)
    elif name == "unreachable_high":
        vf = 0.999
    elif name == "unreachable_low":
        vf = 1e-4
    elif name == "zero":
        dc = np.zeros(n)
    elif name == "uniform":
        rho, dc = np.full(n, 0.3), np.full(n, -0.7)
    elif name == "both_signs":
        col = rng.uniform(-0.2, 1.0, n)
        vf = 0.1
    return rho, dc, dv, col, vf


@pytest.mark.parametrize("n", [1, 7, 300, 40_000])
@pytest.mark.parametrize("name", ["plain", "small", "large", "decades", "unreachable_high", "unreachable_low", "zero",
                                  "uniform", "both_signs"])
def test_filtered_oc_search_is_the_sequential_bisection(cuda_dev, n, name):
    import torch

    from topogpu_b200.context import TopoContext

    rho, dc, dv, col, vf = _case(name, n, np.random.default_rng(n))
    ref, k = sequential(rho, dc, dv, col, vf, 0.2)
    ctx = TopoContext((n, 1, 1), n_levels=1, mode="fp64")
    t = lambda a: torch.tensor(a, device=cuda_dev)  # noqa: E731
    out, ev = ctx.oc_filtered(t(rho), t(dc), t(dv), t(col), vf, 0.2)
    assert ev == k
    assert np.array_equal(out.cpu().numpy(), ref)
    ctx.close()


@pytest.mark.parametrize("nel,rmin", [((1, 1, 1), 0.5), ((2, 3, 1), 2.3), ((5, 4, 70), 3.0), ((7, 9, 33), 1.5), ((3, 2, 2), 5.5)])
def test_filter_rows_cut_on_both_sides(cuda_dev, nel, rmin):
    import torch

    from topogpu_b200.context import TopoContext

    i = np.stack(np.meshgrid(*map(np.arange, nel), indexing="ij"), -1).reshape(-1, 3).astype(float)
    d = np.sqrt(((i[:, None] - i[None]) ** 2).sum(-1))
    W = np.where(d <= rmin - 1e-10, rmin - d, 0.0)
    np.fill_diagonal(W, rmin)
    H = W / W.sum(axis=1, keepdims=True)
    x = np.random.default_rng(2).uniform(0, 1, len(i))
    ctx = TopoContext(nel, n_levels=1, mode="fp64")
    xt = torch.tensor(x, device=cuda_dev)
    np.testing.assert_allclose(ctx.filter(rmin, xt).cpu().numpy(), H @ x, rtol=1e-14)
    np.testing.assert_allclose(ctx.filter(rmin, xt, transpose=True).cpu().numpy(), H.T @ x, rtol=1e-14)
    ctx.close()
