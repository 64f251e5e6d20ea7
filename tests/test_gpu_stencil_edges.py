"""The coarse stencil kernel at node counts inside, at and just past the 32
nodes of a CTA, with one-element extents and more than one run of neighbours
cut off at the ends of the grid.

The spectral bound of a level is ten power iterations with that kernel in
FP64 (Rayleigh quotient of D^-1 K): compared with the same iterations on the
exported level operator in NumPy. Ten products of FP64 sums of 81 terms,
normalised each time: 1e-12 accumulated, held to 1e-10."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nel,levels", [((6, 6, 6), 3), ((14, 6, 6), 3), ((13, 9, 7), 3), ((62, 2, 2), 3), ((9, 3, 20), 3),
                                        ((30, 14, 2), 3), ((2, 2, 62), 3), ((4, 30, 4), 3)])
def test_level_spectral_bound(cuda_dev, nel, levels):
    import torch

    from topogpu_b200.context import TopoContext

    ndof = 3 * int(np.prod([n + 1 for n in nel]))
    mask = np.ones(ndof, dtype=np.uint8)
    mask[: 3 * (nel[1] + 1) * (nel[2] + 1)] = 0
    E = np.random.default_rng(3).uniform(0.05, 1.0, int(np.prod(nel)))
    ctx = TopoContext(nel, n_levels=levels, mode="fp64", smoother="reference")
    ctx.set_problem(torch.tensor(mask, device=cuda_dev), torch.zeros(ndof, dtype=torch.float64, device=cuda_dev))
    ctx.gmg_setup(torch.tensor(E, device=cuda_dev))
    lam = ctx.gmg_info()["lambda_max"]
    dims = nel
    for lv in range(1, levels - 1):
        dims = tuple(max(1, n // 2) for n in dims)
        N = [n + 1 for n in dims]
        nn = int(np.prod(N))
        S = ctx.level_operator(lv).cpu().numpy()
        I = np.arange(nn).reshape(N)
        K = np.zeros((3 * nn, 3 * nn))
        for k in range(27):
            d = (k // 9 - 1, (k // 3) % 3 - 1, k % 3 - 1)
            i = I[tuple(slice(max(0, -x), n - max(0, x)) for x, n in zip(d, N))].ravel()
            j = I[tuple(slice(max(0, x), n - max(0, -x)) for x, n in zip(d, N))].ravel()
            for c in range(3):
                for e in range(3):
                    K[3 * i + c, 3 * j + e] = S[k, c, e, i]
        D = np.diag(K).copy()
        free = D > 1e-12
        D[~free] = 1.0
        v = free / np.linalg.norm(free)
        for _ in range(10):
            Kv = K @ v
            q = (v @ Kv) / (v @ (D * v))
            v = Kv / D * free
            v /= np.linalg.norm(v)
        assert abs(lam[lv] - q) <= 1e-10 * q, (lv, lam[lv], q)
    ctx.close()
