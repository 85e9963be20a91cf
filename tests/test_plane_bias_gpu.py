"""The complex64 plane GEMM's mean error: the truncated partial sums' loss is taken back on average.

Each GEMM would come out 6.4e-8 low (two truncations of a 32-term sum, csrc/plane_gemm.cuh); 6.0e-8 of it is added back.
Tolerance for a transform (two GEMMs) of random fields: 2 x 0.5e-8 left over, and as much again for mantissas that are not
spread evenly and last partial sums that are not full: 4e-8, where the uncorrected transform is 1.3e-7 low.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu

hg = pytest.importorskip('hcipy_gb300')


@pytest.mark.parametrize('n,m', [(512, 200), (1024, 256), (640, 128)])
def test_mean_error_of_a_transform(n, m):
    gi = hg.CartesianGrid(hg.RegularCoords([1 / n] * 2, [n, n], [-0.5 + 0.5 / n] * 2))
    go = hg.CartesianGrid(hg.RegularCoords([1.3] * 2, [m, m], [-0.65 * m] * 2))
    ft = hg.MatrixFourierTransform(gi, go)
    gen = torch.Generator('cuda').manual_seed(n)
    e = torch.randn(2, gi.size, dtype=torch.complex64, device='cuda', generator=gen)
    x, y, u, v = (torch.as_tensor(c, device='cuda') for c in ft._coords)
    ref = torch.exp(-1j * v[:, None] * y) @ e.to(torch.complex128).reshape(2, n, n) @ torch.exp(-1j * x[:, None] * u)
    ref = (ref * ft._w_in_scalar).reshape(2, -1)
    mean = ((ft.forward(e).data - ref) * ref.conj()).real.sum() / (ref.abs()**2).sum()
    assert abs(mean.item()) < 4e-8
