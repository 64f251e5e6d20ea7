"""The reciprocal of the coarsest factorisation's pivots against the division, over
the range in which the factorisation uses it: within one unit in the last place
(hardware start to 2^-19, cubed by the step, and two roundings)."""

import numpy as np
import pytest
import torch

from topogpu_b200 import _lib

pytestmark = pytest.mark.gpu


def _values():
    rng = np.random.default_rng(8)
    lo, hi = np.log(1.001e-290), np.log(0.999e290)
    wide = np.exp(rng.uniform(lo, hi, 400_000))
    ones = rng.uniform(1.0, 2.0, 400_000)
    p = 2.0 ** np.arange(-960, 961)
    # mantissas beside the powers of two and beside the places where the start's 20 bits change
    near = np.concatenate([p, np.nextafter(p, np.inf), np.nextafter(p, 0.0)])
    k = 1.0 + np.arange(0, 2 ** 20, 7) * 2.0 ** -20
    edge = np.concatenate([k, np.nextafter(k, 3.0), np.nextafter(k + 2.0 ** -20, 0.0)])
    return np.concatenate([wide, ones, near, edge])


def test_within_one_ulp_of_the_division(cuda_dev):
    d = _values()
    t = torch.tensor(d, device="cuda")
    r = torch.empty_like(t)
    assert _lib.load().topo_debug_recip(t.numel(), t.data_ptr(), r.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    ref = 1.0 / d
    err = np.abs(r.cpu().numpy() - ref) / np.spacing(ref)
    print(f"largest difference {err.max():.0f} ulp, {np.mean(err > 0):.2%} of the values differ")
    assert np.all(err <= 1.0), (d[err > 1.0][:5], err.max())
