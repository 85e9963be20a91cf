"""float64 FFT lines per CTA: a line's result does not depend on how many lines share its CTA.

One field alone spreads its lines over the SMs (few lines per CTA), a batch of them takes wide groups; both run the same
butterflies on a line.  Tolerance: none.  Sizes: mixed radices with ragged last groups, powers of two, Bluestein.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu

hg = pytest.importorskip('hcipy_gb300')


@pytest.mark.parametrize('n,q', [(360, 1), (250, 1), (96, 2), (153, 1), (256, 2), (211, 1), (31, 1), (2, 1)])
def test_a_field_alone_matches_its_batch(n, q):
    grid = hg.make_pupil_grid(n)
    ft = hg.FastFourierTransform(grid, q=q)
    gen = torch.Generator('cuda').manual_seed(n)
    for op, points in ((ft.forward, grid.size), (ft.backward, ft.output_grid.size)):
        e = torch.randn(48, points, dtype=torch.complex128, device='cuda', generator=gen)
        batch = op(e).data
        for i in (0, 47):
            assert torch.equal(op(e[i].contiguous()).data, batch[i])
