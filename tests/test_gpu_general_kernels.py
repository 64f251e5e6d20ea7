"""The level-0 kernels that take what the parity form does not: a stiffness without
the cube's mirror symmetry (tensor-core and CUDA-core streaming kernels, the block
solve's brick kernel, columns one after another) and z extents beyond its windows.
Every epilogue against a dense sum over the elements, whole solves by their residual
under that sum, the tensor-core kernel's bounded wait, and a stiffness that changes
from context to context on one device. In child processes: the contexts of a device
share one stiffness, and no other context may be open when it changes.

Tolerances: FP64 sums of a few hundred terms to 1e-13, FP32 to 2e-6, BF16 inputs with
FP32 accumulation to 1e-5 (those of the operator tests); a solve's true residual lies
within 2 tol (its recursive one is below tol)."""

from __future__ import annotations

import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

COMMON = r"""
import numpy as np, torch
from test_parity_form import general_stiffness
from oracle import fem
from topogpu_b200 import _lib
from topogpu_b200.context import TopoContext
from topogpu_b200.fem import KE_UNIT

class Case:
    def __init__(self, nel, KE, mode="fp64", levels=1):
        rng = np.random.default_rng(3)
        self.nel, self.KE = nel, KE
        nn = (nel[0] + 1) * (nel[1] + 1) * (nel[2] + 1)
        self.ndof = 3 * nn
        free = rng.uniform(size=(nn, 3)) > (0.1 if levels == 1 else 0.0)
        free[: (nel[1] + 1) * (nel[2] + 1)] = False
        self.mask = free.reshape(-1).astype(np.uint8)
        self.E = rng.uniform(0.3, 1.0, int(np.prod(nel))).astype(np.float32)
        self.ed = fem.edof_table(nel)
        self.rng = rng
        self.ctx = TopoContext(nel, n_levels=levels, mode=mode, KE=KE)
        self.ctx.set_problem(torch.tensor(self.mask, device="cuda"), torch.zeros(self.ndof, dtype=torch.float64, device="cuda"))
    def K(self, u, KE=None):
        y = np.zeros(self.ndof)
        np.add.at(y, self.ed, (np.asarray(u, np.float64)[self.ed] @ (self.KE if KE is None else KE)) * self.E.astype(np.float64)[:, None])
        return y * self.mask
    def vec(self, masked=False):
        v = self.rng.standard_normal(self.ndof).astype(np.float32)
        return v * self.mask if masked else v

def t(a, dt):
    return torch.tensor(np.asarray(a), device="cuda").to(dt)

def rel(a, ref):
    return np.linalg.norm(a.double().cpu().numpy() - ref) / np.linalg.norm(ref)

def epilogues(c, dt, tol, u, ud, KE, **kw):
    # u: device operand; ud: its values in double; every epilogue with KE's product
    E, w = t(c.E, dt), c.K(ud, KE)
    b, r0, x0, dinv = c.vec(), c.vec(True), c.vec(), c.rng.uniform(0.1, 1.0, c.ndof).astype(np.float32)
    m = c.mask
    assert rel(c.ctx.level0_apply(u, E, "store", **kw), w) < tol
    assert rel(c.ctx.level0_apply(u, E, "residual", b=t(b, dt), **kw), (b - w) * m) < tol
    r = t(r0, dt)
    c.ctx.level0_apply(u, E, "rupd", r=r, s=0.7, **kw)
    assert rel(r, (r0 - 0.7 * w) * m) < tol
    r, x, d = t(r0, dt), t(x0, dt), t(0 * x0, dt)
    c.ctx.level0_apply(u, E, "cheb", r=r, x=x, d_out=d, dinv=t(dinv, dt), s=0.7, c1=0.3, c2=1.1, ax=0.9, **kw)
    rr = (r0 - 0.7 * w) * m
    dd = (0.3 * ud + 1.1 * dinv.astype(np.float64) * rr) * m  # (a float times a float32 array would round to float32)
    assert rel(r, rr) < tol and rel(d, dd) < tol and rel(x, x0 + 0.9 * dd) < tol

def solves(c, tol=1e-6):
    ctx = c.ctx
    ctx.gmg_setup(t(c.E, torch.float64))
    B = np.stack([c.vec(True) for _ in range(3)]).astype(np.float64)
    Bt = t(B, torch.float64)
    X = torch.zeros_like(Bt)
    _, rr, ok = ctx.block_pcg(Bt, X, tol=tol, maxiter=400)
    assert ok and max(rr) <= tol
    x = torch.zeros_like(Bt[0])
    _, _, ok = ctx.pcg(Bt[0].contiguous(), x, tol=tol, maxiter=400)
    assert ok
    for u, b in [(x, B[0])] + list(zip(X, B)):
        assert np.linalg.norm(b - c.K(u.cpu().numpy())) <= 2 * tol * np.linalg.norm(b)
    ctx.close()
"""

EPILOGUES = COMMON + r"""
KE = general_stiffness()
Kb = fem.bf16_round(KE.astype(np.float32)).astype(np.float64)
for nel in ((7, 5, 3), (33, 17, 40), (3, 4, 400)):
    c = Case(nel, KE, "mixed")
    u = c.vec(True)
    epilogues(c, torch.float64, 1e-13, t(u, torch.float64), u.astype(np.float64), KE)
    epilogues(c, torch.float32, 2e-6, t(u, torch.float32), u.astype(np.float64), KE)
    ub = fem.bf16_round(u).astype(np.float64)
    if nel[2] < 100:  # BF16-stored u: the tensor-core kernel
        # (the direction c1 u uses the stored, rounded u)
        epilogues(c, torch.float32, 1e-5, t(u, torch.float32).bfloat16(), ub, Kb)
    c.ctx.close()
"""

SOLVES = COMMON + r"""
KE = general_stiffness()
for mode in ("fp64", "fp32", "mixed"):
    solves(Case((24, 12, 6), KE, mode, 2))
    solves(Case((19, 11, 9), KE, mode, 2))
"""

LONG_Z = COMMON + r"""
for nel in ((4, 4, 200), (3, 4, 400)):
    for mode in ("fp64", "fp32"):
        solves(Case(nel, KE_UNIT, mode, 2))
"""

WAIT = COMMON + r"""
lib = _lib.load()
c = Case((24, 12, 6), general_stiffness(), "mixed")
u = t(c.vec(True), torch.float32).bfloat16()
E = t(c.E, torch.float32)
assert lib.topo_debug_tc_wait(1, 1 << 14) == 0
c.ctx.matvec(u, E)
try:
    c.ctx.wait_status()
    raise SystemExit("the timeout was not reported")
except RuntimeError as e:
    assert "timed out" in str(e)
finally:
    lib.topo_debug_tc_wait(0, 0)
Kb = fem.bf16_round(c.KE.astype(np.float32)).astype(np.float64)
assert rel(c.ctx.matvec(u, E), c.K(u.double().cpu().numpy(), Kb)) < 1e-5
c.ctx.wait_status()
c.ctx.close()
"""

CHANGES = COMMON + r"""
def product(KE):
    c = Case((24, 12, 6), KE)
    u = c.vec(True).astype(np.float64)
    y = c.ctx.matvec(t(u, torch.float64), t(c.E, torch.float64))
    assert rel(y, c.K(u)) < 1e-13
    c.ctx.close()
    return y
G = general_stiffness()
a, b = product(KE_UNIT), product(G)
for _ in range(2):
    assert torch.equal(product(KE_UNIT), a) and torch.equal(product(KE_UNIT), a) and torch.equal(product(G), b)
"""


@pytest.mark.parametrize("name", ["EPILOGUES", "SOLVES", "LONG_Z", "WAIT", "CHANGES"])
def test_general_kernels(cuda_dev, name):
    env = {**os.environ, "PYTHONPATH": os.pathsep.join([str(ROOT), str(ROOT / "tests")])}
    r = subprocess.run([sys.executable, "-c", globals()[name] + "\nprint('all ok')"], cwd=ROOT, env=env, capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0 and "all ok" in r.stdout, r.stdout[-2000:] + r.stderr[-4000:]
