"""Plain MFTs on the tensor cores between grids whose weights span many decades, with fields that fall as the weights rise.

Every product of a sum then counts alike, and each has to keep the accuracy that the type gives it.  Tolerances, relative
L2 against float64: those of test_plane_gpu.py (complex64 1e-6, complex128 2e-14), whatever the weights span: the weights
multiply the field before it is cut (one rounding more, 2^-24 or 2^-53), so that the field's planes hold the products'
size and the phases' planes are of modulus 1.
"""
import numpy as np
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu

hg = pytest.importorskip('hcipy_gb300')
from hcipy_gb300 import _lib  # noqa: E402

TOL = {torch.complex64: 1e-6, torch.complex128: 2e-14}


def axis(n, decades, step):
    """A logarithmic axis whose weights span `decades`."""
    x = np.logspace(-decades, 0, n)
    return step * n * (x - x.mean())


@pytest.mark.parametrize('dtype', [torch.complex64, torch.complex128])
@pytest.mark.parametrize('decades', [2, 5, 7, 9])
def test_weights_against_the_inverse_field(decades, dtype):
    gi = hg.CartesianGrid(hg.SeparatedCoords([axis(1100, decades, 1 / 512), axis(260, decades, 1 / 400)]))
    go = hg.CartesianGrid(hg.SeparatedCoords([axis(210, decades, 1.3), axis(333, decades, 1.7)]))
    mft = hg.MatrixFourierTransform(gi, go)
    plan = mft._plan(dtype)
    x, y, u, v = mft._coords
    m1, m2 = np.exp(-1j * v[:, None] * y), np.exp(-1j * x[:, None] * u)
    rng = np.random.default_rng(decades)

    def inverse_field(wa, wb):
        """Random phases over the weights of the axes a (along the rows) and b."""
        e = np.exp(2j * np.pi * rng.uniform(size=(2, len(wb), len(wa)))) / (wb[:, None] * wa)
        e = e / np.abs(e).max()
        return torch.from_numpy(e.reshape(2, -1)).to(dtype).cuda()

    (wx, wy), (wu, wv) = mft._win, mft._wout
    assert np.ptp(np.log10(wx)) > decades - 0.5 and np.ptp(np.log10(wv)) > decades - 0.5
    for direction, code, (wa, wb) in (('forward', _lib.HX_FORWARD, (wx, wy)), ('backward', _lib.HX_BACKWARD, (wu, wv)),
                                      ('adjoint', _lib.HX_ADJOINT, (np.ones_like(wu), np.ones_like(wv)))):
        e = inverse_field(wa, wb)
        assert plan.workspace_bytes(code, 2) > 2 * e.element_size() * gi.shape[0] * 210  # the tensor cores
        w = e.to(torch.complex128).cpu().numpy().reshape(2, len(wb), len(wa))
        if direction == 'forward':
            want = m1 @ (w * wx * wy[:, None]) @ m2
        elif direction == 'backward':
            want = m1.conj().T @ (w * wu * wv[:, None]) @ m2.conj().T / (2 * np.pi)**2
        else:
            want = (m1.conj().T @ w @ m2.conj().T) * wx * wy[:, None]
        got = getattr(mft, direction)(e).numpy()
        if direction == 'adjoint':  # every output by itself: the weights scale them
            got, want = got.reshape(want.shape) / (wx * wy[:, None]), want / (wx * wy[:, None])
        assert rel_err(got, want) < TOL[dtype], direction
