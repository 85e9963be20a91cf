"""The tensor-core form of the plain-precision MFT (complex64 and complex128 plans) against the float64 oracle.

Tolerances, relative L2 (derived from the arithmetic stated in csrc/plane_gemm.cuh):
  complex64 : 22-bit operands (2^-22 per element and operand, 3e-7 for their product), FP32 sums of 64-term partial
              sums (1.5e-7 low at most, roundings of 2^-24 each in blocks): below 1e-6
  complex128: operands at 2^-56 of a row maximum and exact sums, far below 1e-15; what is left is the oracle's own
              rounding, at most 2^-53 sqrt(K) ~ 4e-15 at the lengths here, and two ulp of the phase factors: 2e-14
"""
import numpy as np
import pytest
import torch

from conftest import rel_err
from oracle import fourier as ofourier

pytestmark = pytest.mark.gpu

hg = pytest.importorskip('hcipy_gb300')
from hcipy_gb300 import _lib  # noqa: E402

TOL = {torch.complex64: 1e-6, torch.complex128: 2e-14}


def grids(nx, ny, nu, nv):
    gi = hg.CartesianGrid(hg.RegularCoords([1 / nx, 1 / ny], [nx, ny], [-0.5 + 0.5 / nx, -0.5 + 0.5 / ny]))
    go = hg.CartesianGrid(hg.RegularCoords([1.3, 1.7], [nu, nv], [-0.65 * nu, -0.85 * nv]))
    return gi, go


def fields(batch, n, dtype, seed=0):
    rng = np.random.default_rng(seed)
    e = rng.standard_normal((batch, n)) + 1j * rng.standard_normal((batch, n))
    return torch.from_numpy(e).to(dtype).cuda()


def oracle(mft, e, direction):
    x, y, u, v = mft._coords
    f = {'forward': lambda a: ofourier.mft_forward(a, x, y, u, v, mft.input_grid.weights),
         'backward': lambda a: ofourier.mft_backward(a, x, y, u, v, mft.output_grid.weights),
         'adjoint': lambda a: ofourier.mft_adjoint(a, x, y, u, v, mft.input_grid.weights)}[direction]
    return np.stack([f(a) for a in e.to(torch.complex128).cpu().numpy()])


# (nx, ny, nu, nv, batch): rows and columns around the 128-row and 64- and 32-column tiles, lengths that are not
# multiples of a K step, few tiles over a long K (split K in clusters), many tiles, and stacked fields whose
# boundaries fall inside a tile.
SHAPES = [(512, 129, 127, 1100, 1), (130, 700, 97, 515, 2), (2050, 96, 66, 255, 3), (64, 2048, 640, 65, 1),
          (33, 1025, 1023, 95, 1), (385, 383, 129, 257, 5), (2050, 96, 66, 255, 7)]


@pytest.mark.parametrize('dtype', [torch.complex64, torch.complex128])
@pytest.mark.parametrize('shape', SHAPES)
def test_every_direction_at_tile_edges(shape, dtype):
    gi, go = grids(*shape[:4])
    for schedule in ('latency', 'throughput'):
        mft = hg.MatrixFourierTransform(gi, go, schedule=schedule)
        plan = mft._plan(dtype)
        for direction, n, code in (('forward', gi.size, _lib.HX_FORWARD), ('backward', go.size, _lib.HX_BACKWARD),
                                   ('adjoint', go.size, _lib.HX_ADJOINT)):
            e = fields(shape[4], n, dtype)
            least = shape[4] * shape[1] * shape[2] * e.element_size()
            if _lib.lib().hx_mft_workspace_bytes(plan.handle, code, shape[4]) == least:
                continue  # left to the CUDA cores (too few products), whose error other tests bound
            got = getattr(mft, direction)(e).numpy()
            assert rel_err(got, oracle(mft, e, direction)) < TOL[dtype], (direction, schedule)
        assert plan.status() == 0


@pytest.mark.parametrize('dtype', [torch.complex64, torch.complex128])
def test_epilogues_weights_and_the_least_scratch(dtype):
    """A separated grid with weights of its own, a mask and a Babinet source; with the least scratch that is taken the
    same call runs on the CUDA cores."""
    rng = np.random.default_rng(4)
    gi = hg.CartesianGrid(hg.SeparatedCoords([np.sort(rng.uniform(-0.5, 0.5, 450)), np.linspace(-0.4, 0.5, 300)]))
    go = hg.CartesianGrid(hg.SeparatedCoords([np.linspace(-200, 190, 270), np.sort(rng.uniform(-150, 160, 310))]))
    mft = hg.MatrixFourierTransform(gi, go)
    x, y, u, v = mft._coords
    e, f = fields(2, gi.size, dtype, 1), fields(2, go.size, dtype, 2)
    mask, alpha = fields(1, go.size, dtype, 3)[0], 0.3 - 0.7j
    ref = np.stack([ofourier.mft_forward(a, x, y, u, v, gi.weights) for a in e.to(torch.complex128).cpu().numpy()])
    want = mask.cpu().numpy() * (f.cpu().numpy() - alpha * ref)
    got = mft._run(e, gi, go, _lib.HX_FORWARD, alpha, epilogue=_lib.HX_EPI_BABINET, mask=mask, src=f).numpy()
    assert rel_err(got, want) < TOL[dtype]
    assert rel_err(mft.adjoint(f).numpy(), np.stack([ofourier.mft_adjoint(a, x, y, u, v, gi.weights) for a in
                                                     f.to(torch.complex128).cpu().numpy()])) < TOL[dtype]
    plan, lib = mft._plan(dtype), _lib.lib()
    least = 2 * 270 * 300 * e.element_size()  # the intermediate of two fields
    assert lib.hx_mft_workspace_bytes(plan.handle, _lib.HX_FORWARD, 2) > least
    ws, out = torch.empty(least, dtype=torch.uint8, device='cuda'), torch.empty_like(f)
    before = hg.launch_count()
    _lib.check(lib.hx_mft_execute_ex(plan.handle, _lib.HX_FORWARD, 2, _lib.dptr(e), _lib.dptr(out), 0.3, -0.7,
                                     _lib.HX_EPI_BABINET, _lib.dptr(mask), _lib.dptr(f), _lib.dptr(ws), least,
                                     _lib.stream_handle()))
    assert hg.launch_count() - before == 2  # two products instead of two cuts and two products
    assert rel_err(out.cpu().numpy(), want) < (3e-6 if dtype == torch.complex64 else 2e-14)
    with pytest.raises(ValueError):
        _lib.check(lib.hx_mft_execute(plan.handle, _lib.HX_FORWARD, 2, _lib.dptr(e), _lib.dptr(out), 1.0, 0.0,
                                      _lib.dptr(ws), least - 1, _lib.stream_handle()))


@pytest.mark.parametrize('dtype', [torch.complex64, torch.complex128])
def test_extreme_values(dtype):
    """Rows of very different size, subnormal and near-overflow fields, zeros, and a NaN or an infinity that stays in
    its own field."""
    gi, go = grids(512, 400, 260, 250)
    mft = hg.MatrixFourierTransform(gi, go)
    real = torch.float32 if dtype == torch.complex64 else torch.float64
    e = fields(4, gi.size, dtype, 7)
    rows = torch.logspace(0, -12 if real == torch.float32 else -40, 400, dtype=real, device='cuda')
    e[1] = (e[1].reshape(400, 512) * rows[:, None]).reshape(-1)
    want = oracle(mft, e, 'forward')

    def times_two_to_the(z, k):
        for step in (k // 2, k - k // 2):  # the factor itself may be out of range
            z = np.ldexp(z.real, step) + 1j * np.ldexp(z.imag, step)
        return z

    # powers of two: the smallest outputs are about 2^-9 of their field's inputs, so beside the form's own error
    # 2^-120 (float32) leaves them 2^-20 of their size as spacing, 2^-1030 (float64) 2^-35 and its inputs 2^-44
    small, large, tol = (-120, 105, 2e-6) if real == torch.float32 else (-1030, 1000, 1e-10)
    for k in (0, small, large):
        s = torch.from_numpy(times_two_to_the(e.cpu().numpy().astype(np.complex128), k)).to(dtype).cuda()
        got = times_two_to_the(mft.forward(s).numpy().astype(np.complex128), -k)
        for b in range(4):
            assert rel_err(got[b], want[b]) < (tol if k == small else TOL[dtype]), (k, b)
    assert not mft.forward(torch.zeros_like(e)).data.abs().any()
    for bad in (float('nan'), float('inf')):
        s = e.clone()
        s[2, 12345] = bad
        got = mft.forward(s).data
        assert got[2].isnan().all()
        clean = mft.forward(e).data
        for b in (0, 1, 3):
            assert torch.equal(got[b], clean[b])
