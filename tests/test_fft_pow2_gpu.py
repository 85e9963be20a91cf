"""The register-resident power-of-two lines: every length, one and two dimensions, the Fourier filter's fused column pass,
and both orders of the axes of a padded or cropped transform, against float64.

Tolerance, relative L2: a radix-16 line of N points rounds each value about 2 log2 N times (butterflies and twiddles) at
2^-24, at most 2 sqrt(2 * 2 log2 N) 2^-24 for two transforms of 4096 points and below 1e-6 with the float32 inputs.
"""
import numpy as np
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu

hg = pytest.importorskip('hcipy_gb300')

TOL = 1e-6


def field(rng, *shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)


def regular_grid(*dims):
    return hg.CartesianGrid(hg.RegularCoords([1.0 / d for d in dims], list(dims), [-0.5 + 0.5 / d for d in dims]))


@pytest.mark.parametrize('nx,ny,q', [(128, 128, 2), (256, 100, (1, 2.56)), (512, 1024, 2), (1024, 37, (4, 1)),
                                     (33, 2048, (1, 2)), (1000, 2048, (2.048, 1)), (2048, 130, (2, 256 / 130))])
def test_filter_columns_of_every_length(nx, ny, q):
    rng = np.random.default_rng(nx + ny)
    grid = regular_grid(nx, ny)
    ff = hg.FourierFilter(grid, None, q)
    N, c = ff._N, ff._c
    tf = field(rng, N[1], N[0])
    ff.transfer_function = hg.Field(torch.from_numpy(tf.reshape(-1)).cuda(), ff.internal_grid)
    e = field(rng, 2, ny, nx)
    centred = np.fft.ifftshift(tf.astype(np.complex128))
    for direction, t in (('forward', centred), ('backward', centred.conj())):
        pad = np.zeros((2, N[1], N[0]), np.complex128)
        pad[:, c[1]:c[1] + ny, c[0]:c[0] + nx] = e
        want = np.fft.ifft2(np.fft.fft2(pad) * t)[:, c[1]:c[1] + ny, c[0]:c[0] + nx]
        got = getattr(ff, direction)(torch.from_numpy(e.reshape(2, -1)).cuda()).numpy()
        assert rel_err(got, want) < TOL, direction


@pytest.mark.parametrize('n', [256, 512, 1024, 2048, 4096])
def test_filter_in_one_dimension(n):
    rng = np.random.default_rng(n)
    grid = hg.CartesianGrid(hg.RegularCoords([1.0], [n], [0.0]))
    tf = field(rng, n)
    ff = hg.FourierFilter(grid, hg.Field(torch.from_numpy(tf).cuda(), None), 1)
    e = field(rng, 3, n)
    want = np.fft.ifft(np.fft.fft(e.astype(np.complex128)) * np.fft.ifftshift(tf.astype(np.complex128)))
    assert rel_err(ff.forward(torch.from_numpy(e).cuda()).numpy(), want) < TOL


@pytest.mark.parametrize('dims,q,fov', [((64, 1024), 4, 1), ((1024, 64), 4, 1), ((300, 512), (1, 8), (1, 0.25)),
                                        ((512, 300), (8, 1), (0.1, 1)), ((1, 700), (256, 1), 1)])
@pytest.mark.parametrize('dtype', [np.complex64, np.complex128])
def test_either_order_of_the_axes(dims, q, fov, dtype):
    """Padding one axis far more than the other, and cropping: columns first or rows first, in both directions."""
    from oracle import fourier as ofourier
    from oracle.grids import RegularGrid
    rng = np.random.default_rng(dims[0])
    grid = regular_grid(*dims)
    ft = hg.FastFourierTransform(grid, q, fov)
    plan = ofourier.FFTPlan(RegularGrid(grid.delta, grid.dims, grid.zero), q, fov)
    e = field(rng, 2, grid.size).astype(dtype)
    f = field(rng, 2, ft.output_grid.size).astype(dtype)
    tol = TOL if dtype == np.complex64 else 1e-12
    for b in range(2):
        assert rel_err(ft.forward(torch.from_numpy(e).cuda()).numpy()[b], plan.forward(e[b].astype(complex))) < tol
        assert rel_err(ft.backward(torch.from_numpy(f).cuda()).numpy()[b], plan.backward(f[b].astype(complex))) < tol
