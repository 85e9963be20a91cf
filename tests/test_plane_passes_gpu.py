"""Batches of the plain MFT whose scratch is taken in several passes: results written over the inputs, as in one pass.

Tolerance: none, a field's result does not depend on the others of its pass.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu

hg = pytest.importorskip('hcipy_gb300')
from hcipy_gb300 import _lib  # noqa: E402


@pytest.mark.parametrize('n,m', [(256, 300), (300, 256)])  # fields that grow and fields that shrink
def test_results_over_the_inputs(n, m):
    batch = 2500  # 2 MB of scratch each, 4 GB to a pass
    gi = hg.CartesianGrid(hg.RegularCoords([1 / n] * 2, [n, n], [-0.5 + 0.5 / n] * 2))
    go = hg.CartesianGrid(hg.RegularCoords([1.3] * 2, [m, m], [-0.65 * m] * 2))
    ft = hg.MatrixFourierTransform(gi, go)
    e = torch.randn(batch, gi.size, dtype=torch.complex64, device='cuda', generator=torch.Generator('cuda').manual_seed(3))
    plan, lib = ft._plan(torch.complex64), _lib.lib()
    need = plan.workspace_bytes(_lib.HX_FORWARD, batch)
    ws = torch.empty(need, dtype=torch.uint8, device='cuda')

    def run(src, dst):
        before = hg.launch_count()
        _lib.check(lib.hx_mft_execute(plan.handle, _lib.HX_FORWARD, batch, _lib.dptr(src), _lib.dptr(dst), 1.0, 0.0,
                                      _lib.dptr(ws), need, _lib.stream_handle()))
        assert hg.launch_count() - before > 4  # more passes than one

    want = torch.empty(batch, go.size, dtype=torch.complex64, device='cuda')
    run(e, want)
    shared = torch.empty(batch * max(gi.size, go.size), dtype=torch.complex64, device='cuda')
    shared[:e.numel()] = e.reshape(-1)
    run(shared, shared)
    assert torch.equal(shared[:want.numel()], want.reshape(-1))
