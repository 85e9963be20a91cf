"""A padded FFT with scratch for the rows-first order of its axes alone, where it takes the columns first given more.

Both orders compute the same sums of products in other groupings; tolerance: 2e-6 of the norm in complex64 (that of the FFT
tests), 1e-13 in complex128.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu

hg = pytest.importorskip('hcipy_gb300')
from hcipy_gb300 import _lib  # noqa: E402


@pytest.mark.parametrize('dtype', [torch.complex64, torch.complex128])
@pytest.mark.parametrize('batch', [1, 3])
def test_scratch_of_the_rows_first_order(dtype, batch):
    nx, ny = 100, 10
    gi = hg.CartesianGrid(hg.RegularCoords([1 / nx, 1 / ny], [nx, ny], [-0.5, -0.5]))
    ft = hg.FastFourierTransform(gi, q=[2, 2.1])
    mx, my = ft.output_grid.dims
    e = torch.randn(batch, gi.size, dtype=dtype, device='cuda', generator=torch.Generator('cuda').manual_seed(0))
    want = ft.forward(e).data
    lib, plan = _lib.lib(), ft._plan(dtype)
    rows_first = batch * ny * int(mx) * e.element_size()
    assert batch * int(my) * nx * e.element_size() == lib.hx_fft_workspace_bytes(plan.handle, _lib.HX_FORWARD, batch) > rows_first
    ws = torch.full((rows_first + 256,), 0x5a, dtype=torch.uint8, device='cuda')
    out = torch.empty_like(want)

    def run(nbytes):
        _lib.check(lib.hx_fft_execute(plan.handle, _lib.HX_FORWARD, batch, _lib.dptr(e), _lib.dptr(out), _lib.dptr(ws),
                                      nbytes, _lib.stream_handle()))

    run(rows_first)
    assert ((out - want).norm() / want.norm()).item() < (2e-6 if dtype == torch.complex64 else 1e-13)
    assert (ws[rows_first:] == 0x5a).all()
    with pytest.raises(ValueError):
        run(rows_first - 1)
