"""Which kernel runs the level-0 operator of a mesh (host rule, no GPU): the parity
form on every ordinary mesh, the general kernels where a window would be little more
than its halo row or the windows just miss a wave. The time of either side is
measured beside the rule; the meshes below are those measurements."""

from __future__ import annotations

import ctypes as C
import math
import random

import pytest

from topogpu_b200 import _lib

PARITY, TENSOR, STREAM, BRICK = range(4)
STORE, RESIDUAL, CHEB, DOT, RUPD = range(5)


def route(nel, dtype, epi):
    k = C.c_int(-1)
    assert _lib.load().topo_debug_route(*nel, dtype, epi, 148, C.byref(k)) == 0
    return k.value


@pytest.mark.parametrize("nel, dtype, epi, kernel", [
    # FP64 Chebyshev step: 115 us against 224, 114 against 115; 207 against 123, 206 against 115
    ((80, 125, 100), _lib.F64, CHEB, PARITY), ((80, 80, 155), _lib.F64, CHEB, PARITY),
    ((80, 73, 170), _lib.F64, CHEB, BRICK), ((80, 67, 185), _lib.F64, CHEB, BRICK),
    # FP64 product: 54 us against 78 to 83
    ((80, 73, 170), _lib.F64, STORE, PARITY), ((80, 67, 185), _lib.F64, DOT, PARITY),
    # FP32: 49.5 us against 62 (step: 62 against 62); 91 against 61 (110 against 62)
    ((80, 40, 310), _lib.F32, STORE, PARITY), ((80, 40, 310), _lib.F32, CHEB, PARITY),
    ((80, 36, 340), _lib.F32, STORE, BRICK), ((80, 33, 371), _lib.F32, CHEB, BRICK),
    ((80, 62, 200), _lib.F32, CHEB, PARITY),
    # BF16 with FP32 u
    ((80, 40, 310), _lib.BF16_F32IN, CHEB, PARITY), ((80, 36, 340), _lib.BF16_F32IN, CHEB, BRICK),
    ((80, 69, 180), _lib.BF16_F32IN, CHEB, PARITY),
    # small: 16.8 us against 14.6; 9.5 against 27; 10.3 against 8.6
    ((24, 13, 185), _lib.F64, CHEB, BRICK), ((24, 7, 340), _lib.F32, STORE, PARITY), ((24, 7, 340), _lib.BF16, STORE, BRICK),
    # BF16 product: 37 us against 39, 37 against 35
    ((80, 80, 155), _lib.BF16, STORE, PARITY), ((80, 73, 170), _lib.BF16, STORE, TENSOR), ((80, 73, 170), _lib.BF16, CHEB, PARITY),
    # z beyond every window
    ((80, 62, 200), _lib.F64, STORE, BRICK), ((3, 4, 400), _lib.F32, STORE, STREAM), ((4, 4, 2000), _lib.F32, STORE, BRICK),
])
def test_measured_meshes(nel, dtype, epi, kernel):
    assert route(nel, dtype, epi) == kernel


def test_ordinary_meshes_run_the_parity_form():
    rng = random.Random(4)
    for _ in range(2000):
        nx = int(round(math.exp(rng.uniform(math.log(2), math.log(200)))))
        nel = (nx, max(1, int(nx * rng.uniform(0.3, 0.6))), max(1, int(nx * rng.uniform(0.15, 0.5))))
        for dtype in (_lib.F64, _lib.F32, _lib.BF16, _lib.BF16_F32IN):
            for epi in (STORE, RESIDUAL, CHEB, RUPD):
                assert route(nel, dtype, epi) == PARITY, (nel, dtype, epi)
