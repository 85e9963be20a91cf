"""Scratch of the plain MFT that starts at any address its elements may have: the same results, nothing written outside."""
import pytest
import torch

pytestmark = pytest.mark.gpu

hg = pytest.importorskip('hcipy_gb300')
from hcipy_gb300 import _lib  # noqa: E402


@pytest.mark.parametrize('dtype,offset', [(torch.complex64, 8), (torch.complex64, 248), (torch.complex128, 16),
                                          (torch.complex128, 240)])
def test_scratch_at_an_offset(dtype, offset):
    n, m = 640, 130
    gi = hg.CartesianGrid(hg.RegularCoords([1 / n] * 2, [n, n], [-0.5 + 0.5 / n] * 2))
    go = hg.CartesianGrid(hg.RegularCoords([1.3] * 2, [m, m], [-0.65 * m] * 2))
    ft = hg.MatrixFourierTransform(gi, go)
    e = torch.randn(2, gi.size, dtype=dtype, device='cuda', generator=torch.Generator('cuda').manual_seed(2))
    plan, lib = ft._plan(dtype), _lib.lib()
    need = plan.workspace_bytes(_lib.HX_FORWARD, 2)
    ws = torch.full((need + 1024,), 0x5a, dtype=torch.uint8, device='cuda')
    out = torch.empty(2, go.size, dtype=dtype, device='cuda')
    before = hg.launch_count()
    _lib.check(lib.hx_mft_execute(plan.handle, _lib.HX_FORWARD, 2, _lib.dptr(e), _lib.dptr(out), ft._w_in_scalar, 0.0,
                                  _lib.dptr(ws) + offset, need, _lib.stream_handle()))
    assert hg.launch_count() - before == 4  # on the tensor cores
    assert torch.equal(out, ft.forward(e).data)
    assert (ws[:offset] == 0x5a).all() and (ws[offset + need:] == 0x5a).all()
