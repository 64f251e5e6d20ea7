"""The level-0 operator in parity form (csrc/kmatvec_pt.cu).

CPU: the rule that selects it. In the basis of sums and differences of the
corner values (one 2x2x2 Hadamard transform per component) the cube's
stiffness couples only values of one parity class, and so do its FP32 and
BF16 roundings; a stiffness without the mirror symmetry does not pass.

GPU: every precision against the oracle on meshes at the edges of the
kernel's windows (31 elements per warp, one and several windows, the last
z extent a window takes and the first it does not, one-element extents), and
the general kernels through a context with a stiffness that has no mirror
symmetry. Tolerances: FP64 sums of a few hundred terms to 1e-13, FP32 to 2e-6
(the operator tests' bound), BF16 inputs with FP32 accumulation to 1e-5.
"""

from __future__ import annotations

import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT
from oracle import fem
from topogpu_b200.fem import KE_UNIT

CORNERS = np.array([[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0], [0, 0, 1], [1, 0, 1], [1, 1, 1], [0, 1, 1]])


def class_coupling(KE):
    """(largest entry between different classes, largest entry) of H KE H^T / 64."""
    s = 2.0 * CORNERS - 1.0
    par = [(px, py, pz) for px in (0, 1) for py in (0, 1) for pz in (0, 1)]
    H = np.array([[np.prod(s[a] ** np.array(p)) for a in range(8)] for p in par])
    K = np.einsum("pa,aibj,qb->piqj", H, KE.reshape(8, 3, 8, 3), H) / 64.0
    cls = np.array([[tuple(np.array(p) ^ np.eye(3, dtype=int)[c]) for c in range(3)] for p in par])
    same = (cls[:, :, None, None, :] == cls[None, None, :, :, :]).all(axis=-1)
    return np.abs(K[~same]).max(), np.abs(K).max()


@pytest.mark.parametrize("KE", [KE_UNIT, fem.hex8_stiffness(), KE_UNIT.astype(np.float32).astype(np.float64),
                                fem.bf16_round(KE_UNIT.astype(np.float32)).astype(np.float64)])
def test_cube_stiffness_couples_one_class_only(KE):
    cross, top = class_coupling(KE)
    assert cross <= 1e-12 * top


def general_stiffness():
    """Symmetric positive semidefinite, translations in its null space, no mirror symmetry."""
    rng = np.random.default_rng(5)
    B = rng.standard_normal((24, 24))
    P = np.eye(24) - np.kron(np.full((8, 8), 0.125), np.eye(3))
    return KE_UNIT + 0.05 * P @ B @ B.T @ P / 24.0


def test_general_stiffness_is_not_taken():
    cross, top = class_coupling(general_stiffness())
    assert cross > 1e-4 * top


MESHES = [(1, 1, 1), (2, 1, 3), (1, 30, 2), (3, 2, 29), (5, 3, 30), (4, 5, 61), (6, 9, 40), (150, 2, 2), (9, 46, 17),
          (3, 61, 92), (2, 2, 185), (2, 2, 186), (2, 2, 278), (2, 2, 279), (2, 3, 371), (2, 3, 372)]


@pytest.mark.gpu
@pytest.mark.parametrize("nel", MESHES)
def test_operator_at_window_edges(cuda_dev, nel):
    import torch

    from topogpu_b200.context import TopoContext

    rng = np.random.default_rng(int(np.prod(nel)))
    ndof = 3 * (nel[0] + 1) * (nel[1] + 1) * (nel[2] + 1)
    mask = (rng.uniform(size=ndof) > 0.1).astype(np.uint8)
    u = rng.standard_normal(ndof) * mask
    E = rng.uniform(1e-3, 1.0, int(np.prod(nel)))
    ctx = TopoContext(nel, n_levels=1, mode="mixed")
    t = lambda a, dt: torch.tensor(a, device=cuda_dev).to(dt)  # noqa: E731
    ctx.set_problem(torch.tensor(mask, device=cuda_dev), torch.zeros(ndof, dtype=torch.float64, device=cuda_dev))
    ref = fem.matvec_full(u, E, nel) * mask
    nrm = np.linalg.norm(ref)
    y64 = ctx.matvec(t(u, torch.float64), t(E, torch.float64)).cpu().numpy()
    assert np.linalg.norm(y64 - ref) <= 1e-13 * nrm
    u32, E32 = u.astype(np.float32), E.astype(np.float32)
    ref32 = fem.matvec_full(u32.astype(np.float64), E32.astype(np.float64), nel) * mask
    y32 = ctx.matvec(t(u32, torch.float32), t(E32, torch.float32)).cpu().numpy()
    assert np.linalg.norm(y32 - ref32) <= 2e-6 * nrm
    emu = fem.matvec_full(fem.bf16_round(u32), E32, nel, "bf16").astype(np.float64) * mask
    yb = ctx.level0_apply(t(u32, torch.float32), t(E32, torch.float32), "store", u_fp32_to_bf16=True).cpu().numpy()
    assert np.linalg.norm(yb - emu) <= 1e-5 * np.linalg.norm(emu)
    for y in (y64, y32, yb):
        assert np.all(y[mask == 0] == 0.0)
    ctx.close()


GENERAL = r"""
import numpy as np, torch
from test_parity_form import general_stiffness
from oracle import fem
from topogpu_b200.context import TopoContext
KE = general_stiffness()
for nel in ((7, 5, 3), (33, 17, 40), (3, 4, 400)):
    rng = np.random.default_rng(3)
    n = int(np.prod(nel)); ndof = 3 * (nel[0] + 1) * (nel[1] + 1) * (nel[2] + 1)
    mask = (rng.uniform(size=ndof) > 0.1).astype(np.uint8)
    u = (rng.standard_normal(ndof) * mask).astype(np.float32); E = rng.uniform(1e-3, 1.0, n).astype(np.float32)
    b = rng.standard_normal(ndof).astype(np.float32)
    ed = fem.edof_table(nel)
    def ref(uu, K):
        y = np.zeros(ndof); np.add.at(y, ed, (uu.astype(np.float64)[ed] @ K) * E.astype(np.float64)[:, None]); return y * mask
    ctx = TopoContext(nel, n_levels=1, mode="mixed", KE=KE)
    t = lambda a, dt=torch.float32: torch.tensor(np.asarray(a), device="cuda").to(dt)
    ctx.set_problem(torch.tensor(mask, device="cuda"), torch.zeros(ndof, dtype=torch.float64, device="cuda"))
    rel = lambda a, c: np.linalg.norm(a.double().cpu().numpy() - c) / np.linalg.norm(c)
    assert rel(ctx.matvec(t(u, torch.float64), t(E, torch.float64)), ref(u, KE)) < 1e-13
    assert rel(ctx.matvec(t(u), t(E)), ref(u, KE)) < 2e-6
    ub, Kb = fem.bf16_round(u), fem.bf16_round(KE.astype(np.float32)).astype(np.float64)
    assert rel(ctx.matvec(t(u).bfloat16(), t(E)), ref(ub, Kb)) < 1e-5
    w, r, x, d = ref(ub, Kb), t(b * mask), t(b), t(0 * b)
    dinv = rng.uniform(0.1, 1.0, ndof).astype(np.float32)
    ctx.level0_apply(t(u), t(E), "cheb", r=r, x=x, d_out=d, dinv=t(dinv), s=0.7, c1=0.3, c2=1.1, ax=0.9, u_fp32_to_bf16=True)
    rr = (b - 0.7 * w) * mask; dd = (0.3 * u + 1.1 * dinv * rr) * mask
    assert rel(r, rr) < 1e-5 and rel(d, dd) < 1e-5 and rel(x, b + 0.9 * dd) < 1e-5
    y = ctx.level0_apply(t(u), t(E), "residual", b=t(b))
    assert rel(y, (b - ref(u, KE)) * mask) < 2e-6
    ctx.close()
print("general ok")
"""


@pytest.mark.gpu
def test_general_stiffness_runs_the_general_kernels(cuda_dev):
    """In a child process: contexts of one device share one stiffness."""
    env = {**os.environ, "PYTHONPATH": os.pathsep.join([str(ROOT), str(ROOT / "tests")])}
    r = subprocess.run([sys.executable, "-c", GENERAL], cwd=ROOT, env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and "general ok" in r.stdout, r.stdout[-2000:] + r.stderr[-4000:]
