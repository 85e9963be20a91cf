"""The complex64 MFT on the tensor cores, whatever the field.

Fields of random values, of real or imaginary values alone, smooth ones, and single pixels (whose sums have one term, so
that nothing averages out).

Operands in digits (sums of up to 128 terms, and the forward direction up to 960 points a side): the error of each sum is that
of one FP32 rounding, for sums of 16, 32 and 96 terms, of a K' whose halves hold an odd number of 32s, and of many
partial sums.
Tolerance, relative L2 against float64, 1e-7.  A transform rounds three times to 24 bits (the two sums and the product with
the grid's weight): a rounding is 2^-24 at most, uniform, of a value whose mantissa is spread over its logarithm, 2.5e-8
in the mean square, so 4.4e-8 together.  The operands are exact, or cut at 2^-29 of a row's maximum at most, 2^-29 / sqrt(3) =
1.1e-9 of it in the mean square: 5e-9 of random values.  The products of digits that are left out are 2.5e-9 of the two maxima
in the mean square: 1.2e-8 of random values.
With mantissas that are not spread evenly (all pixels of a smooth field alike) a rounding may be 3.4e-8 in
the mean square: 7e-8 in all.
Mean error (a factor on the whole transform), 4e-8: roundings to nearest have none for random fields; where
all sums are alike they share one, 2^-25 = 3e-8 at most in the mean.

Operands in floating planes (grids of more than 960 points a side): 3e-7.  Two operands of each of two products are rounded by
2^-23 at most, 6.9e-8 in the mean square, 1.4e-7 together; the factor that takes the truncated sums' loss back is 2^-23 too
large for sums that have lost nothing, 2.4e-7 in both products if each falls on it: 2.8e-7.  With the second product in
digits (the other directions up to 960 points): 1e-7 and 1.2e-7 of the first, and 7e-8: 1.7e-7, tolerance 2e-7.  Real
and imaginary fields have the same mean error: as many of their partial sums have that factor.  Tolerance: 1e-8, where
one partial sum more of five is 2.4e-8.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu

hg = pytest.importorskip('hcipy_gb300')


def field_of(kind, batch, size, seed):
    gen = torch.Generator('cuda').manual_seed(seed)
    e = torch.randn(batch, size, dtype=torch.complex64, device='cuda', generator=gen)
    if kind == 'real':
        return torch.complex(e.real, torch.zeros_like(e.real))
    if kind == 'imaginary':
        return torch.complex(torch.zeros_like(e.real), e.imag)
    if kind == 'smooth':
        return torch.polar(torch.ones_like(e.real), (6 * torch.rand(batch, 1, device='cuda', generator=gen)).expand(e.shape))
    if 'pixel' in kind:
        at = torch.randint(0, size, (batch, 1), device='cuda', generator=gen)
        return torch.zeros_like(e).scatter_(1, at, torch.ones_like(e) if kind == 'unit pixel' else e.gather(1, at))
    return e


def errors(n, m, batch, kind, adjoint=False):
    """Relative error and mean error of the transform of n^2 points to m^2, or of its adjoint from m^2 points to n^2."""
    gi = hg.CartesianGrid(hg.RegularCoords([1 / n] * 2, [n, n], [-0.5 + 0.5 / n] * 2))
    go = hg.CartesianGrid(hg.RegularCoords([1.3] * 2, [m, m], [-0.65 * m] * 2))
    ft = hg.MatrixFourierTransform(gi, go)
    e = field_of(kind, batch, (go if adjoint else gi).size, n)
    x, y, u, v = (torch.as_tensor(c, device='cuda') for c in ft._coords)
    m1, m2 = torch.exp(-1j * v[:, None] * y), torch.exp(-1j * x[:, None] * u)
    ft._plan(torch.complex64)
    before = hg.launch_count()
    if adjoint:
        ref, got = m1.T.conj() @ e.to(torch.complex128).reshape(batch, m, m) @ m2.T.conj(), ft.adjoint(e).data
    else:
        ref, got = m1 @ e.to(torch.complex128).reshape(batch, n, n) @ m2, ft.forward(e).data
    assert hg.launch_count() - before == 4  # the tensor cores
    ref = (ref * ft._w_in_scalar).reshape(batch, -1)
    d = got - ref
    return (d.norm() / ref.norm()).item(), ((d * ref.conj()).real.sum() / (ref.abs()**2).sum()).item()


KINDS = ['random', 'real', 'imaginary', 'smooth', 'pixel', 'unit pixel']


@pytest.mark.parametrize('kind', KINDS)
@pytest.mark.parametrize('n,m,batch', [(16, 700, 64), (32, 1000, 64), (96, 600, 16), (160, 600, 16), (640, 130, 4), (960, 257, 1)])
def test_digits(n, m, batch, kind):
    error, mean = errors(n, m, batch, kind)
    assert error < 1e-7
    assert abs(mean) < 4e-8


@pytest.mark.parametrize('kind', KINDS)
@pytest.mark.parametrize('n,m,batch', [(600, 160, 16), (130, 640, 4), (257, 960, 1)])
def test_second_product_in_digits(n, m, batch, kind):
    assert errors(n, m, batch, kind, adjoint=True)[0] < 2e-7


@pytest.mark.parametrize('kind', KINDS)
@pytest.mark.parametrize('n,m,batch', [(160, 1000, 16), (961, 200, 4), (2048, 257, 1)])
def test_floating_planes(n, m, batch, kind):
    assert errors(n, m, batch, kind)[0] < 3e-7


def test_floating_planes_of_real_and_imaginary_fields():
    assert abs(errors(160, 1000, 16, 'real')[1] - errors(160, 1000, 16, 'imaginary')[1]) < 1e-8
