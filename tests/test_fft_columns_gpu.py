"""4096-point columns in pairs and in fours per CTA (pairs up to two columns per SM), odd counts among them, against float64.

Tolerance: that of test_fft_pow2_gpu.py, 1e-6 of the norm.
"""
import numpy as np
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu

hg = pytest.importorskip('hcipy_gb300')


@pytest.mark.parametrize('nx,batch', [(5, 1), (75, 4), (301, 1), (303, 1), (304, 1), (305, 1), (320, 1), (125, 3)])
def test_columns(nx, batch):
    ny, q = 1024, 4
    gi = hg.CartesianGrid(hg.RegularCoords([1 / nx, 1 / ny], [nx, ny], [0.0, 0.0]))
    ft = hg.FastFourierTransform(gi, q=[1, q])
    e = torch.randn(batch, gi.size, dtype=torch.complex64, device='cuda', generator=torch.Generator('cuda').manual_seed(nx))
    x, y = (torch.as_tensor(c, device='cuda') for c in gi.separated_coords)
    u, v = (torch.as_tensor(c, device='cuda') for c in ft.output_grid.separated_coords)
    m1, m2 = torch.exp(-1j * v[:, None] * y), torch.exp(-1j * x[:, None] * u)
    want = (m1 @ e.to(torch.complex128).reshape(batch, ny, nx) @ m2 * gi.weights).reshape(batch, -1)
    got = ft.forward(e)
    assert rel_err(got.numpy(), want.cpu().numpy()) < 1e-6
    assert rel_err(ft.backward(got).numpy(), e.cpu().numpy()) < 2e-6  # two transforms
    assert np.isfinite(got.numpy()).all()
