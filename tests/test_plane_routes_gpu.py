"""Which plain transforms the tensor cores take: small ones with long sums (complex64), all but the smallest (complex128).

The tensor-core results against float64.  Tolerances: complex64 5e-7 (operands of 22 bits of their row's maximum, 2^-22 = 2.4e-7, and FP32 sums of
32 terms), complex128 5e-15 (the reference itself sums up to 1001 terms in float64).
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

hg = pytest.importorskip('hcipy_gb300')


@pytest.mark.parametrize('n_in,n_out,batch,dtype,launches', [
    ((1001, 501), (33, 33), 1, torch.complex64, 4),
    ((310, 290), (20, 16), 9, torch.complex64, 4),    # sums of 600 terms
    ((310, 289), (20, 16), 9, torch.complex64, 2),    # of 599
    ((50, 50), (50, 50), 1, torch.complex128, 4),
    ((64, 64), (32, 32), 16, torch.complex128, 4),
    ((16, 16), (16, 17), 9, torch.complex128, 2),     # 7.8e4 products
    ((41, 36), (34, 18), 9, torch.complex128, 4),
])
def test_small_forward_transforms(n_in, n_out, batch, dtype, launches):
    from hcipy_gb300 import _lib
    gi, go = (hg.CartesianGrid(hg.RegularCoords(d, n, -(np.asarray(n) - 1) / 2 * d))
              for n, d in ((n_in, 1 / 64), (n_out, 0.37)))
    ft = hg.MatrixFourierTransform(gi, go)
    gen = torch.Generator('cuda').manual_seed(3)
    e = torch.randn(batch, gi.size, dtype=dtype, device='cuda', generator=gen)
    ft.forward(e)
    before = _lib.launch_count()
    got = ft.forward(e).data
    assert _lib.launch_count() - before == launches
    if launches != 4:
        return  # the CUDA cores, whose error other tests bound
    x, y, u, v = (torch.as_tensor(c, device='cuda') for c in ft._coords)
    ref = torch.exp(-1j * v[:, None] * y) @ e.to(torch.complex128).reshape(batch, y.numel(), x.numel()) \
        @ torch.exp(-1j * x[:, None] * u) * ft._w_in_scalar
    err = (got - ref.reshape(batch, -1)).norm() / ref.norm()
    assert err < (5e-7 if dtype == torch.complex64 else 5e-15)
