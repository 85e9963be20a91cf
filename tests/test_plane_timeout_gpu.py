"""A bounded wait of the plain tensor-core GEMM that runs out: NaN in the result, and the plan's status.

HX_FAULT=wait gives the waits 10 ms and leaves out the loads of one CTA per tile (the first of those that share the tile's
sum, or the only one).  No copy is in flight then, and every wait ends by its limit, so the kernels return.  The CTAs of
a cluster that are not stalled themselves must not finish sums that lack a part.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu

hg = pytest.importorskip('hcipy_gb300')


def grid(n, delta):
    return hg.CartesianGrid(hg.RegularCoords([delta] * 2, [n, n], [-(n - 1) / 2 * delta] * 2))


@pytest.mark.parametrize('schedule', ['latency', 'throughput'])  # a K split in clusters where it pays, and none
@pytest.mark.parametrize('dtype', [torch.complex64, torch.complex128])
def test_a_wait_that_runs_out_leaves_nan(dtype, schedule, monkeypatch):
    gi, go = grid(700, 1 / 700), grid(130, 1.3)
    ft = hg.MatrixFourierTransform(gi, go, schedule=schedule)
    e = torch.randn(gi.size, dtype=dtype, device='cuda', generator=torch.Generator('cuda').manual_seed(1))
    good = ft.forward(e).data.clone()
    plan = ft._plan(dtype)
    assert torch.isfinite(good.abs()).all() and plan.status() == 0
    monkeypatch.setenv('HX_FAULT', 'wait')
    bad = ft.forward(e).data
    monkeypatch.delenv('HX_FAULT')
    assert bad.isnan().all()
    assert plan.status() == -4  # HX_ERR_TIMEOUT
    assert plan.status() == 0
    assert torch.equal(ft.forward(e).data, good)
    assert plan.status() == 0
