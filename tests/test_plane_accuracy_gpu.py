"""The complex64 MFT on the tensor cores: the error of each sum is that of one FP32 rounding, whatever the field.

Fields of random values, of real or imaginary values alone, smooth ones, and single pixels (whose sums have one term, so
that nothing averages out), for sums of 16, 32 and 96 terms, of a K' whose halves hold an odd number of 32s, and of many
partial sums.

Tolerance, relative L2 against float64, 1e-7.  A transform rounds three times to 24 bits (the two sums and the product with
the grid's weight): a rounding is 2^-24 at most, uniform, of a value whose mantissa is spread over its logarithm, 2.5e-8
in the mean square, so 4.4e-8 together.  The operands, cut at 2^-27 of a row's maximum at most, add 2^-27 / sqrt(3) = 4.3e-9
of that maximum twice per product, about 2e-8 of random values (maximum 4 to 5 times the mean square), in both products:
5e-8 in all.  With mantissas that are not spread evenly (all pixels of a smooth field alike) a rounding may be 3.4e-8 in
the mean square: 7e-8.
Mean error (a factor on the whole transform), 4e-8: roundings to nearest have none for random fields; where
all sums are alike they share one, 2^-25 = 3e-8 at most in the mean.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu

hg = pytest.importorskip('hcipy_gb300')
from hcipy_gb300 import _lib  # noqa: E402


@pytest.mark.parametrize('kind', ['random', 'real', 'imaginary', 'smooth', 'pixel', 'unit pixel'])
@pytest.mark.parametrize('n,m,batch', [(16, 700, 64), (32, 700, 64), (96, 600, 16), (160, 600, 16), (640, 130, 4),
                                       (2048, 257, 1)])
def test_error_of_a_transform(n, m, batch, kind):
    gi = hg.CartesianGrid(hg.RegularCoords([1 / n] * 2, [n, n], [-0.5 + 0.5 / n] * 2))
    go = hg.CartesianGrid(hg.RegularCoords([1.3] * 2, [m, m], [-0.65 * m] * 2))
    ft = hg.MatrixFourierTransform(gi, go)
    assert ft._plan(torch.complex64).workspace_bytes(_lib.HX_FORWARD, batch) > batch * n * m * 8  # the tensor cores
    gen = torch.Generator('cuda').manual_seed(n)
    e = torch.randn(batch, gi.size, dtype=torch.complex64, device='cuda', generator=gen)
    if kind == 'real':
        e = torch.complex(e.real, torch.zeros_like(e.real))
    elif kind == 'imaginary':
        e = torch.complex(torch.zeros_like(e.real), e.imag)
    elif kind == 'smooth':
        e = torch.polar(torch.ones_like(e.real), (6 * torch.rand(batch, 1, device='cuda', generator=gen)).expand(e.shape))
    elif 'pixel' in kind:
        at = torch.randint(0, gi.size, (batch, 1), device='cuda', generator=gen)
        e = torch.zeros_like(e).scatter_(1, at, torch.ones_like(e) if kind == 'unit pixel' else e.gather(1, at))
    x, y, u, v = (torch.as_tensor(c, device='cuda') for c in ft._coords)
    ref = torch.exp(-1j * v[:, None] * y) @ e.to(torch.complex128).reshape(batch, n, n) @ torch.exp(-1j * x[:, None] * u)
    ref = (ref * ft._w_in_scalar).reshape(batch, -1)
    d = ft.forward(e).data - ref
    assert (d.norm() / ref.norm()).item() < 1e-7
    assert abs(((d * ref.conj()).real.sum() / (ref.abs()**2).sum()).item()) < 4e-8
