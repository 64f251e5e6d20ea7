"""The parity-class blocks of the element stiffness that K.u multiplies with are
the exact sums rounded once: an error of their own would show in every FP64 result
(sums in double are off by up to 3.4 units in the last place)."""

from __future__ import annotations

import ctypes as C
from fractions import Fraction

import numpy as np
import pytest

from oracle import fem
from test_parity_form import CORNERS, general_stiffness
from topogpu_b200 import _lib
from topogpu_b200.fem import KE_UNIT


def _blocks(KE):
    KE = np.ascontiguousarray(KE, dtype=np.float64)
    out = np.empty(72)
    sym = C.c_int(-1)
    assert _lib.load().topo_debug_class_blocks(KE.ctypes.data, out.ctypes.data, C.byref(sym)) == 0
    return out.reshape(8, 3, 3), bool(sym.value)


def _exact(KE):
    h = [[(-1) ** sum(((p >> (2 - d)) & 1) and not CORNERS[a][d] for d in range(3)) for a in range(8)] for p in range(8)]
    F = [[Fraction(float(v)) for v in row] for row in KE]
    e = (4, 2, 1)
    return [[[sum(h[q ^ e[c]][a] * h[q ^ e[d]][b] * F[3 * a + c][3 * b + d] for a in range(8) for b in range(8)) / 64
              for d in range(3)] for c in range(3)] for q in range(8)]


@pytest.mark.parametrize("KE", [KE_UNIT, fem.hex8_stiffness(), fem.hex8_stiffness(0.123, 7.0),
                                KE_UNIT.astype(np.float32).astype(np.float64),
                                fem.bf16_round(KE_UNIT.astype(np.float32)).astype(np.float64)])
def test_blocks_are_rounded_once(KE):
    got, sym = _blocks(KE)
    assert sym
    # one rounding to double, and 6 additions with 64 bits of mantissa over 64 entries
    slack = Fraction(6 * 64 * float(np.abs(KE).max())) / 2 ** 64 / 64
    for q, blk in enumerate(_exact(KE)):
        for c in range(3):
            for d in range(3):
                x = blk[c][d]
                assert abs(Fraction(float(got[q, c, d])) - x) <= abs(x) / 2 ** 53 + slack, (q, c, d)


def test_a_stiffness_without_the_symmetry_is_told():
    assert not _blocks(general_stiffness())[1]
    assert not _blocks(np.full((24, 24), np.nan))[1]
