"""The fused dot product of the level-0 operator leaves one partial sum per CTA: a
context's buffer holds all of them on every mesh, thin and very wide ones too."""

from __future__ import annotations

import ctypes as C

import pytest

from topogpu_b200 import _lib


def _query(nel, f64, nsm=148):
    blocks, room = C.c_longlong(), C.c_longlong()
    assert _lib.load().topo_debug_reduction(*nel, int(f64), nsm, C.byref(blocks), C.byref(room)) == 0
    return blocks.value, room.value


@pytest.mark.parametrize("nel, f64", [
    ((1, 262_300, 185), True),    # 62 nodes per window: more windows than 2^18
    ((1, 87_500, 371), False),
    ((3, 30_000, 4_000), True),   # no window layout: bricks
    ((160, 80, 80), True),
    ((160, 80, 80), False),
    ((1, 1, 1), True),
])
def test_partial_sums_fit(nel, f64):
    blocks, room = _query(nel, f64)
    assert 1 <= blocks <= room


def test_wide_meshes_need_more_than_the_usual_buffer():
    usual = 1 << 18
    for nel, f64 in (((1, 262_300, 185), True), ((1, 87_500, 371), False), ((3, 30_000, 4_000), True)):
        blocks, room = _query(nel, f64)
        assert blocks > usual and room >= blocks
    assert _query((160, 80, 80), True)[1] == usual
