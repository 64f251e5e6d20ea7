"""R.A.P in one-dimensional passes on extents where the transfers change form:
one element, odd extents (the last fine node has one parent), one and two
coarse elements. Every level operator against P^T K P formed with the oracle's
assembled matrix and the row-normalised trilinear prolongation: a few hundred
FP64 products per entry, 1e-12 of the largest entry."""

from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sp



pytestmark = pytest.mark.gpu


def prolong_1d(nf):
    nc = max(1, nf // 2)
    P = np.zeros((nf + 1, nc + 1))
    for i in range(nf + 1):
        par = [i // 2] if i % 2 == 0 else [j for j in (i // 2, i // 2 + 1) if j <= nc]
        P[i, par] = 1.0 / len(par)
    return sp.csr_matrix(P), nc


@pytest.mark.parametrize("nel", [(8, 4, 2), (12, 6, 4), (13, 9, 7), (16, 3, 5), (9, 1, 6), (20, 2, 1)])
def test_level_operators(cuda_dev, nel):
    import torch

    from topogpu_b200.context import TopoContext

    levels = 4
    rng = np.random.default_rng(7)
    E = rng.uniform(0.05, 1.0, int(np.prod(nel)))
    ndof = 3 * int(np.prod([n + 1 for n in nel]))
    mask = np.ones(ndof, dtype=np.uint8)
    mask[: 3 * (nel[1] + 1) * (nel[2] + 1)] = 0
    ctx = TopoContext(nel, n_levels=levels, mode="fp64")
    ctx.set_problem(torch.tensor(mask, device=cuda_dev), torch.zeros(ndof, dtype=torch.float64, device=cuda_dev))
    ctx.gmg_setup(torch.tensor(E, device=cuda_dev))
    ops = [ctx.level_operator(lv).cpu().numpy() for lv in range(1, levels)]
    dims = nel
    for lv in range(1, levels):
        if lv > 1:
            Ps, nc = zip(*(prolong_1d(n) for n in dims))
            P = sp.kron(sp.kron(sp.kron(Ps[0], Ps[1]), Ps[2]), sp.eye(3)).tocsr()
            ref = (P.T @ A @ P).toarray() * np.outer(m_next, m_next)
            dims = nc
        else:
            dims = tuple(max(1, n // 2) for n in nel)
        S = ops[lv - 1]
        N = [n + 1 for n in dims]
        nn = int(np.prod(N))
        I = np.arange(nn).reshape(N)
        A = np.zeros((3 * nn, 3 * nn))
        for k in range(27):
            d = (k // 9 - 1, (k // 3) % 3 - 1, k % 3 - 1)
            src = tuple(slice(max(0, -x), n - max(0, x)) for x, n in zip(d, N))
            dst = tuple(slice(max(0, x), n - max(0, -x)) for x, n in zip(d, N))
            i, j = I[src].ravel(), I[dst].ravel()
            for c in range(3):
                for e in range(3):
                    A[3 * i + c, 3 * j + e] = S[k, c, e, i]
        if lv > 1:
            assert np.abs(A - ref).max() <= 1e-12 * np.abs(ref).max(), lv
        # the next level's free set by injection of this level's linear index
        m_here = mask if lv == 1 else m_next
        if lv == 1:
            m_here = inject(mask, nel, dims)
        nd = tuple(max(1, n // 2) for n in dims)
        m_next = inject(m_here, dims, nd)
        A = sp.csr_matrix(A)
    ctx.close()


def inject(m, f, c):
    out = np.zeros(3 * int(np.prod([n + 1 for n in c])), dtype=np.uint8)
    q = 0
    for I in range(c[0] + 1):
        for J in range(c[1] + 1):
            for K in range(c[2] + 1):
                fn = (2 * I * (f[1] + 1) + 2 * J) * (f[2] + 1) + 2 * K
                for d in range(3):
                    out[q] = m[3 * fn + d] if 3 * fn + d < len(m) else 0
                    q += 1
    return out
