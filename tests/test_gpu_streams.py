"""One context called from several streams: the library orders the calls among
themselves, whatever stream each comes from, and its own buffers, those made by
a first call among them, are ready on the stream that uses them."""

import pytest
import torch

pytestmark = pytest.mark.gpu

NEL, LEVELS = (43, 21, 17), 3


def _solver():
    from topogpu_b200.state import StateSolver

    nx, ny, nz = NEL
    nn = (nx + 1) * (ny + 1) * (nz + 1)
    free = torch.ones(nn, 3, dtype=torch.uint8)
    free[: (ny + 1) * (nz + 1)] = 0  # the face x = 0
    F = torch.zeros(nn, 3, dtype=torch.float64)
    F[-1, 2] = -1.0
    return StateSolver(NEL, free.reshape(-1).numpy(), F.reshape(-1).numpy(), precision="fp64", n_levels=LEVELS,
                       warm_start=False, tol=1e-8)


def _inputs(s):
    g = torch.Generator().manual_seed(11)
    n = s.ctx.n_elem
    rho = (0.3 + 0.4 * torch.rand(n, generator=g, dtype=torch.float64)).cuda()
    dc = -(0.1 + torch.rand(n, generator=g, dtype=torch.float64)).cuda()
    dv = (0.5 + torch.rand(n, generator=g, dtype=torch.float64)).cuda()
    r = torch.randn(s.ctx.ndof, generator=g, dtype=torch.float64).cuda() * s.free_mask
    B = torch.randn(3, s.ctx.ndof, generator=g, dtype=torch.float64).cuda() * s.free_mask
    return rho, dc, dv, r, B


def _first_calls(s, rho, dc, dv, B):
    out, evals = s.ctx.oc_projected(2.0, rho, dc, dv, 8.0, 0.5, 0.4, 0.2)
    c, U = s.solve_block(rho, B)
    return out, evals, c, U


def test_first_calls_beside_a_busy_default_stream():
    ref = _solver()
    rho, dc, dv, _, B = _inputs(ref)
    o0, e0, c0, U0 = _first_calls(ref, rho, dc, dv, B)
    torch.cuda.synchronize()
    s = _solver()
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    torch.cuda._sleep(200_000_000)  # about 0.1 s of work on the default stream
    with torch.cuda.stream(side):
        o, e, c, U = _first_calls(s, rho, dc, dv, B)
    torch.cuda.synchronize()
    assert e == e0 and torch.equal(o, o0)
    assert c == c0 and torch.equal(U, U0)
    s.close()
    ref.close()


def test_calls_alternate_between_streams():
    s = _solver()
    ctx = s.ctx
    rho, dc, dv, r, _ = _inputs(s)
    E = ctx.modulus(rho, 3.0, 1.0, 1e-9)
    ctx.gmg_setup(E)
    calls = [lambda: ctx.matvec(r, E), lambda: ctx.filter(2.0, rho), lambda: ctx.gmg_apply(r),
             lambda: ctx.oc(rho, dc, 0.4, 0.2)[0], lambda: ctx.filter(2.0, dc, transpose=True),
             lambda: ctx.oc_projected(2.0, rho, dc, dv, 8.0, 0.5, 0.4, 0.2)[0]]
    want = [f().clone() for f in calls]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.current_stream()]
    for turn in range(20):
        got = []
        for i, f in enumerate(calls):
            with torch.cuda.stream(streams[(i + turn) % 3]):
                got.append(f())
        torch.cuda.synchronize()
        for i, (a, b) in enumerate(zip(got, want)):
            assert torch.equal(a, b), (turn, i)
    s.close()


def test_a_captured_call_leaves_the_order_of_the_others():
    s = _solver()
    ctx = s.ctx
    rho, _, _, r, _ = _inputs(s)
    E = ctx.modulus(rho, 3.0, 1.0, 1e-9)
    y0 = ctx.matvec(r, E)
    ctx.gmg_setup(E)  # the last call before the capture ran on the context's stream
    op0 = ctx.level_operator(1)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        op = ctx.level_operator(1)
    with torch.cuda.stream(torch.cuda.Stream()):
        y = ctx.matvec(r, E)  # waits for the set-up, not for the captured copy
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, y0) and torch.equal(op, op0)
    s.close()
