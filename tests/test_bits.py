"""Outputs whose roundings must not change (tests/golden/make_bits.py): FP16
wave fields, where a changed last bit of the FP32 arithmetic flips stored
values, boundary-saving gradients under a free surface, whose adjoint amplifies
it, and the forms of the free surface and of the absorbing layers on every
kind of rows.  Bit for bit."""
import os

import numpy as np
import pytest

from tests.golden.make_bits import CASES, run

GOLDEN = os.path.join(os.path.dirname(__file__), "golden", "bits.npz")


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(CASES))
def test_same_bits(name, cuda_device):
    stored = np.load(GOLDEN)
    want = {k.split("/")[1]: stored[k] for k in stored.files if k.split("/")[0] == name}
    got = run(name)
    assert got.keys() == want.keys() and np.abs(want["vx0"]).max() > 0
    for k in want:
        assert np.array_equal(got[k], want[k]), (k, int((got[k] != want[k]).sum()), float(np.abs(got[k] - want[k]).max()))
