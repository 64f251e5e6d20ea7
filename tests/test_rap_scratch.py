"""R.A.P's intermediate operators take a bounded part of the device's memory: the
passes run slab by slab of x planes where the whole would be larger, with the bits
of the whole."""

from __future__ import annotations

import ctypes as C

import pytest

from topogpu_b200 import _lib


@pytest.mark.parametrize("nel", [(160, 80, 80), (640, 640, 640), (2000, 300, 300), (400, 20, 3000), (3, 40, 50), (1, 1, 1)])
def test_scratch_is_bounded(nel):
    n = C.c_longlong(0)
    assert _lib.load().topo_debug_rap_room(*nel, C.byref(n)) == 0
    x, y, z = (max(1, v // 2) + 1 for v in nel)  # level 1's nodes
    cy, cz = (max(1, max(1, v // 2) // 2) + 1 for v in nel[1:])
    plane = 243 * (y + cy) * cz
    # three planes or 512 MB, whichever is more; never more than the whole
    assert n.value <= max(3 * plane, 1 << 26)
    assert n.value == x * plane if x * plane <= 1 << 26 else n.value >= 3 * plane


@pytest.mark.gpu
@pytest.mark.parametrize("nel, levels", [((13, 9, 7), 4), ((16, 3, 5), 4), ((9, 1, 6), 4), ((24, 12, 6), 4), ((31, 6, 9), 4),
                                         ((4, 5, 4), 3), ((6, 5, 4), 3)])
def test_slabs_have_the_bits_of_the_whole(nel, levels):
    import torch

    from topogpu_b200.context import TopoContext

    ctx = TopoContext(nel, n_levels=levels, mode="fp64")
    g = torch.Generator().manual_seed(5)
    mask = torch.ones(ctx.ndof, dtype=torch.uint8)
    mask[: 3 * (nel[1] + 1) * (nel[2] + 1)] = 0
    ctx.set_problem(mask.cuda(), torch.zeros(ctx.ndof, dtype=torch.float64, device="cuda"))
    E = (0.05 + torch.rand(ctx.n_elem, generator=g, dtype=torch.float64)).cuda()
    ctx.gmg_setup(E)
    want = [ctx.level_operator(lv).clone() for lv in range(2, levels)]
    for planes in (3, 4, 5, 8):  # one, two and three planes of the coarse grid at a time
        assert ctx._lib.topo_debug_scratch(ctx._h, planes) == 0
        ctx.gmg_setup(E)
        for lv, w in enumerate(want, 2):
            assert torch.equal(ctx.level_operator(lv), w), (planes, lv)
    ctx.close()
