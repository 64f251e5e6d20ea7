"""A bounded wait that runs out inside a solve or a set-up is reported by that call,
not by a later one: the test hook withholds the first plane's copy of the level-0
K.u, whose kernels then give up, raise the flag and exit."""

import pytest
import torch

from topogpu_b200 import _lib

pytestmark = pytest.mark.gpu


def _ctx(mode):
    from topogpu_b200.context import TopoContext

    nel = (24, 12, 6)
    ctx = TopoContext(nel, n_levels=2, mode=mode)
    mask = torch.ones(nel[0] + 1, nel[1] + 1, nel[2] + 1, 3, dtype=torch.uint8)
    mask[0] = 0
    mask = mask.reshape(-1).cuda()
    g = torch.Generator().manual_seed(2)
    E = (0.5 + torch.rand(ctx.n_elem, generator=g, dtype=torch.float64)).cuda()
    B = torch.randn(3, ctx.ndof, generator=g, dtype=torch.float64).cuda() * mask
    ctx.set_problem(mask, B[0].contiguous())
    return ctx, E, B


# (the mixed mode's spectral bound runs the general kernel, which the hook leaves alone)
@pytest.mark.parametrize("mode,call", [(m, c) for m in ("fp64", "fp32", "mixed") for c in ("setup", "block", "fgmres")
                                       if (m, c) != ("mixed", "setup")])
def test_timeout_is_reported_by_the_call(mode, call):
    lib = _lib.load()
    ctx, E, B = _ctx(mode)
    run = {
        "setup": lambda: ctx.gmg_setup(E),
        "block": lambda: ctx.block_pcg(B, torch.zeros_like(B), tol=1e-6, maxiter=200),
        "fgmres": lambda: ctx.fgmres(B[0].contiguous(), torch.zeros_like(B[0]), tol=1e-6, maxiter=200),
    }[call]
    ctx.gmg_setup(E * (0.5 if call == "setup" else 1.0))  # (set-up: new moduli, so that the bounds are estimated)
    assert call == "setup" or run()[2]
    torch.cuda.synchronize()
    assert lib.topo_debug_tc_wait(1, 1 << 14) == 0
    try:
        with pytest.raises(RuntimeError, match="wait timed out"):
            run()
        torch.cuda.synchronize()
    finally:
        lib.topo_debug_tc_wait(0, 0)
    try:  # (launches behind the one that was reported may have raised the flag again)
        ctx.wait_status()
    except RuntimeError:
        pass
    ctx.gmg_setup(E)
    X = torch.zeros_like(B)
    _, rr, ok = ctx.block_pcg(B, X, tol=1e-6, maxiter=200)
    assert ok and max(rr) <= 1e-6
    ctx.wait_status()
    ctx.close()
