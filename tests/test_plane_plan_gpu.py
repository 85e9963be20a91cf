"""Plans of the plain MFT: which of their transforms have a tensor-core form, and what a failure of its operands does.

No memory for the cut operands leaves the plan to the CUDA cores; any other failure is the plan's own (it is not passed
over for a form that takes ten times as long).
"""
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu

hg = pytest.importorskip('hcipy_gb300')


def grids(nx, ny, nu, nv):
    gi = hg.CartesianGrid(hg.RegularCoords([1 / nx, 1 / ny], [nx, ny], [-0.5 + 0.5 / nx, -0.5 + 0.5 / ny]))
    go = hg.CartesianGrid(hg.RegularCoords([1.3, 1.7], [nu, nv], [-0.65 * nu, -0.85 * nv]))
    return gi, go


def on_tensor_cores(mft, dtype, direction, batch):
    """Four launches (two cuts and two products) rather than one or two."""
    e = torch.zeros((batch, (mft.input_grid if direction == 'forward' else mft.output_grid).size), dtype=dtype, device='cuda')
    mft._plan(dtype)
    before = hg.launch_count()
    getattr(mft, direction)(e)
    return hg.launch_count() - before == 4


@pytest.mark.parametrize('shape,batch,c64', [
    ((512, 129, 127, 1100), 1, (True, True)), ((130, 700, 97, 515), 2, (True, True)), ((2050, 96, 66, 255), 3, (True, True)),
    ((64, 2048, 640, 65), 1, (True, True)), ((33, 1025, 1023, 95), 1, (True, True)), ((385, 383, 129, 257), 5, (True, True)),
    ((256, 256, 128, 128), 1, (False, False)), ((15, 900, 900, 900), 1, None), ((8193, 64, 64, 64), 1, None)])
def test_the_path_of_each_direction(shape, batch, c64):
    """complex64: 6e7 complex multiply-adds or 600 terms in the two sums; complex128: 1e5.  None: no planes at all."""
    mft = hg.MatrixFourierTransform(*grids(*shape))
    forward, back = c64 or (False, False)
    for direction, want in (('forward', forward), ('backward', back), ('adjoint', back)):
        assert on_tensor_cores(mft, torch.complex64, direction, batch) == want, direction
        assert on_tensor_cores(mft, torch.complex128, direction, batch) == (c64 is not None)


@pytest.mark.parametrize('dtype', [torch.complex64, torch.complex128])
def test_failures_of_the_operands(dtype, monkeypatch):
    gi, go = grids(700, 640, 130, 97)
    e = torch.randn(gi.size, dtype=dtype, device='cuda', generator=torch.Generator('cuda').manual_seed(1))
    full = hg.MatrixFourierTransform(gi, go)
    assert on_tensor_cores(full, dtype, 'forward', 1)
    monkeypatch.setenv('HX_FAULT', 'operand_memory')
    plain = hg.MatrixFourierTransform(gi, go)
    plain._plan(dtype)
    monkeypatch.delenv('HX_FAULT')
    assert not on_tensor_cores(plain, dtype, 'forward', 1)
    before = hg.launch_count()
    got = plain.forward(e).numpy()
    assert hg.launch_count() - before == 2  # two products, no cuts
    # the CUDA cores' FP32 sums of 700 terms (test_plane_gpu.py), or float64
    assert rel_err(got, full.forward(e).numpy()) < (3e-6 if dtype == torch.complex64 else 2e-14)
    monkeypatch.setenv('HX_FAULT', 'operand_map')
    with pytest.raises(hg.HXError):
        hg.MatrixFourierTransform(gi, go)._plan(dtype)
    monkeypatch.delenv('HX_FAULT')
    assert torch.equal(hg.MatrixFourierTransform(gi, go).forward(e).data, full.forward(e).data)
