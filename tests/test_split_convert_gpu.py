"""The split transform's float-float -> float64 conversion: the integer form against the float64 addition.

A field times a power of two (or times -1) has slices that differ in their scale alone, so its split transform is the
same times that power, whichever way a value's conversion takes: the integer sum for magnitudes above 2^-75, the float64
addition below.  Tolerance: none where the low parts of the results stay normal floats; for the smallest scale their
last bits fall under 2^-149, an absolute error of a few 2^-149 before the scale is taken out.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

hg = pytest.importorskip('hcipy_gb300')


@pytest.mark.parametrize('n_in,n_out', [(96, 64), (130, 33)])
@pytest.mark.parametrize('exponent,sign', [(0, -1), (30, 1), (-40, -1), (-66, 1)])
def test_power_of_two_scales_are_exact(n_in, n_out, exponent, sign):
    rng = np.random.default_rng(11)
    xg = (np.arange(n_in) - n_in / 2 + 0.5) / n_in
    ug = (np.arange(n_out) - n_out / 2 + 0.5) * 0.41
    gi = hg.CartesianGrid(hg.RegularCoords(1.0 / n_in, [n_in, n_in], [xg[0], xg[0]]))
    go = hg.CartesianGrid(hg.RegularCoords(0.41, [n_out, n_out], [ug[0], ug[0]]))
    e = torch.from_numpy(rng.standard_normal((3, gi.size)) + 1j * rng.standard_normal((3, gi.size)))
    e[1] = 0
    split = hg.MatrixFourierTransform(gi, go, precision='split')
    ref = split.forward(e.cuda()).numpy()
    got = split.forward((e * (sign * 2.0 ** exponent)).cuda()).numpy()
    assert ref.dtype == np.complex128
    assert not np.any(ref[1]) and np.all(ref[0] != 0)
    err = np.abs((got * (sign * 2.0 ** -exponent) - ref).view(np.float64)).max()
    assert err <= (8 * 2.0 ** (-149 - exponent) if exponent < -60 else 0.0)
