"""The persistent split GEMM (more output tiles than SMs) against the one with a CTA per tile: the same bits.

A batch of fields makes enough tiles for the persistent kernel; one of its fields alone does not, and with the
throughput schedule neither splits K, so both sum the same products in the same order.  Tolerance: none.  The shapes
have neighbouring column tiles that share A (an even number), row tiles that share B, and neither; fields that begin
within a tile and within a warp's rows; ragged rows and columns; one shape has rows of an odd length, whose
intermediate field keeps the other kernel.  Not-a-numbers and infinities of one field stay in that field.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

hg = pytest.importorskip('hcipy_gb300')


def grid(n, delta):
    n = np.asarray(n)
    return hg.CartesianGrid(hg.RegularCoords(delta, n, -(n - 1) / 2 * delta))


@pytest.mark.parametrize('n_in,n_out', [((66, 70), (124, 70)), ((124, 50), (128, 60)), ((250, 47), (60, 130)),
                                        ((65, 64), (123, 129))])
@pytest.mark.parametrize('masked', [False, True])
def test_batches_match_single_fields(n_in, n_out, masked):
    from hcipy_gb300 import _lib
    batch = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    gi, go = grid(n_in, 1 / 64), grid(n_out, 0.37)
    ft = hg.MatrixFourierTransform(gi, go, precision='split', schedule='throughput')
    gen = torch.Generator('cuda').manual_seed(5)

    def fields(n, dtype):
        return torch.randn(batch, n, dtype=dtype, device='cuda', generator=gen)

    def run(e, src, dst, direction, alpha, mask):
        epi = {} if mask is None else {'epilogue': _lib.HX_EPI_MUL, 'mask': mask}
        return ft._run(e, src, dst, direction, alpha, **epi).data.cpu().numpy()

    for src, dst, direction, dtype, alpha in ((gi, go, _lib.HX_FORWARD, torch.complex64, 0.3 + 0j),
                                              (gi, go, _lib.HX_FORWARD, torch.complex128, -0.7j),
                                              (go, gi, _lib.HX_BACKWARD, torch.complex64, 1 + 0j),
                                              (go, gi, _lib.HX_ADJOINT, torch.complex128, 0.2 - 0.9j)):
        e = fields(src.size, dtype)
        e[3, 17] = float('nan')
        e[batch - 2, 5] = float('inf')
        mask = fields(dst.size, torch.complex64)[0] if masked else None
        if masked:
            mask[::2] = mask[::2].real.to(torch.complex64)
        got = run(e, src, dst, direction, alpha, mask)
        for i in (0, 1, 3, 4, batch // 2, batch - 2, batch - 1):
            np.testing.assert_array_equal(got[i], run(e[i:i + 1], src, dst, direction, alpha, mask)[0])
            assert np.all(np.isfinite(got[i])) or i in (3, batch - 2)
    assert ft._plan(torch.complex64).status() == 0
