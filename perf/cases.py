"""The work that users of hcipy_gb300 have it do, as cases that can be timed and compared.

Every case goes through the operator API as a user's program calls it: the elements (propagators, coronagraphs, the
deformable mirror, the transforms) are built once in ``prepare`` and kept, ``run`` is one pass on new fields.  Lengths
are in units of the pupil diameter and the wavelength unless a case says otherwise.  ``exact`` states the same
physics in float64 with dense Fourier matrices, numpy.fft or torch.fft, and torch's autograd.
"""
import math

import numpy as np
import torch

import hcipy_gb300 as hg

DEVICE = 'cuda'
COMPLEX = {'c64': torch.complex64, 'c128': torch.complex128}
SIZE = {'c64': 8, 'c128': 16}


def listed():
    return [
        # The smallest call: a 256^2 pupil imaged by a lens, the reference's CPU-sized propagation.
        _lens('lens-256-c64', 256, 4, 16, 'c64'),
        # The type that numpy gives a user who does not ask for one: complex128 fields through a lens.
        _lens('lens-512-c128', 512, 4, 32, 'c128'),
        # Back from a focal plane to an odd-sized pupil, a few fields at a time (ragged in every dimension).
        _lens('lens-1001-c64-back', 1001, 3, 27.5, 'c64', batch=3, backward=True),
        # The plain Lyot coronagraph and its image, four fields stacked (wavefronts of a time series).
        _lyot('lyot-1024-c64', 1024, 8, 32, 4, 32, 'c64', 'fp32', 4),
        # The benchmark's workload: 2048^2 pupil, 512^2 focal-plane mask, 512^2 image, split precision.
        _lyot('lyot-2048-split', 2048, 8, 32, 8, 32, 'c64', 'split', 1),
        # One gradient step of a dark-hole optimisation: 64 command vectors of a 34 x 34 deformable mirror.
        {'name': 'gradient-512-split', 'kind': 'gradient', 'n': 512, 'actuators': 34, 'vectors': 64,
         'precision': 'split'},
        # A vortex coronagraph with its nested focal grids, in the default complex128.
        {'name': 'vortex-256-c128', 'kind': 'vortex', 'n': 256, 'charge': 2, 'dtype': 'c128'},
        # A broadband frame: 21 wavelengths on their own focal grids, recorded once and replayed for each field.
        {'name': 'broadband-1024-split', 'kind': 'broadband', 'n': 1024, 'wavelengths': 21, 'precision': 'split'},
        # The zero-padded FFT to a full, finely sampled focal plane.
        _fft('fft-1024-c64', 1024, 4, 1.0, 'c64'),
        # Back from a cropped FFT plane, a length with factors 3 and 5, complex128.
        _fft('fft-360-c128-back', 360, 2, 0.5, 'c128', backward=True),
        # Free-space propagation of a turbulent telescope pupil.
        {'name': 'asp-1024-c64', 'kind': 'asp', 'n': 1024, 'distance': 5.0, 'dtype': 'c64', 'backward': False},
        # A frozen-flow frame: a phase screen moved by a fraction of a pixel and applied to a field.
        {'name': 'screen-1023-c64', 'kind': 'screen', 'n': 1023, 'dtype': 'c64'},
    ]


def _lens(name, n, q, airy, dtype, batch=1, backward=False, precision='fp32'):
    return {'name': name, 'kind': 'lens', 'n': n, 'q': q, 'airy': airy, 'dtype': dtype, 'batch': batch,
            'backward': backward, 'precision': precision}


def _lyot(name, n, q, airy, image_q, image_airy, dtype, precision, batch):
    return {'name': name, 'kind': 'lyot', 'n': n, 'q': q, 'airy': airy, 'image_q': image_q,
            'image_airy': image_airy, 'dtype': dtype, 'precision': precision, 'batch': batch}


def _fft(name, n, q, fov, dtype, backward=False):
    return {'name': name, 'kind': 'fft', 'n': n, 'q': q, 'fov': fov, 'dtype': dtype, 'backward': backward}


def draw(rng):
    """One more case of the same ranges: sizes over their logarithm, odd ones among them."""
    def size(lo, hi):
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        kind = rng.random()
        if kind < 0.3:  # a power of two, as most programs choose
            return max(lo, min(hi, 1 << int(round(math.log2(n)))))
        return n | 1 if kind < 0.6 and (n | 1) <= hi else n

    kind = rng.choice(['lens', 'lens', 'lens', 'lyot', 'lyot', 'gradient', 'vortex', 'broadband', 'fft', 'fft', 'asp',
                       'asp', 'screen'])
    dtype = rng.choice(['c64', 'c64', 'c128'])
    if kind == 'lens':
        c = _lens('', size(96, 1536 if dtype == 'c64' else 768), rng.choice([2, 3, 4, 6]),
                  rng.choice([8.0, 12.5, 16.0, 24.0, 32.0]), dtype, rng.choice([1, 1, 2, 5]), rng.random() < 0.4,
                  rng.choice(['fp32', 'fp32', 'split']))
    elif kind == 'lyot':
        c = _lyot('', size(192, 1400 if dtype == 'c64' else 512), rng.choice([4, 8]), rng.choice([16, 24, 32]),
                  rng.choice([3, 4, 8]), rng.choice([16, 20.5, 32]), dtype, rng.choice(['fp32', 'split']),
                  rng.choice([1, 2, 4]))
    elif kind == 'gradient':
        c = {'kind': kind, 'n': size(128, 512), 'actuators': rng.randint(10, 34), 'vectors': rng.choice([1, 8, 31, 64]),
             'precision': rng.choice(['fp32', 'split'])}
    elif kind == 'vortex':
        c = {'kind': kind, 'n': size(64, 320) & ~1, 'charge': rng.choice([2, 4, 6]), 'dtype': dtype}
    elif kind == 'broadband':
        c = {'kind': kind, 'n': size(256, 1024), 'wavelengths': rng.randint(3, 21),
             'precision': rng.choice(['fp32', 'split'])}
    elif kind == 'fft':
        q = rng.choice([1, 2, 4])
        most = 4096 if dtype == 'c64' else 2048
        c = _fft('', size(100, min(1024, most // q)), q, rng.choice([1.0, 1.0, 0.5, 0.3]), dtype, rng.random() < 0.5)
    elif kind == 'asp':
        c = {'kind': kind, 'n': size(100, 1024), 'distance': round(rng.uniform(0.5, 50.0), 2), 'dtype': dtype,
             'backward': rng.random() < 0.5}
    else:
        c = {'kind': kind, 'n': size(200, 2048), 'dtype': dtype}
    c.pop('name', None)
    return c


# ---- inputs, from the seed alone ------------------------------------------------------------------------------


def _axis(n):
    """The centres of n pixels across a diameter of 1."""
    return (np.arange(n) - (n - 1) / 2) / n


def _focal_axis(q, airy):
    """The coordinates, in lambda/D, of a focal grid with q samples for each lambda/D out to `airy` of them."""
    m = int(2 * q * airy)
    return (np.arange(m) - m // 2) / q


def _dev(a):
    return torch.as_tensor(np.asarray(a), device=DEVICE)


def _disk(n, diameter):
    x = _dev(_axis(n))
    return (x[None, :]**2 + x[:, None]**2 <= (diameter / 2)**2).double()


def _phases(n, batch, seed, rms):
    """Smooth random phases (batch, n, n): two dozen waves with amplitudes that fall with their frequency."""
    rng = np.random.default_rng(seed)
    x = _dev(_axis(n))
    out = torch.zeros((batch, n, n), dtype=torch.float64, device=DEVICE)
    for b in range(batch):
        for _ in range(24):
            kx, ky = rng.integers(-6, 7, 2)
            a = rng.standard_normal() / (1 + math.hypot(kx, ky))
            p = rng.uniform(0, 2 * math.pi)
            out[b] += a * torch.cos(2 * math.pi * (kx * x[None, :] + ky * x[:, None]) + p)
    return out * (rms / out.std())


def _pupil_fields(n, batch, seed, dtype, rms=0.3):
    """Aberrated circular pupils, flat (batch, n^2), or (n^2,) for one."""
    e = torch.polar(_disk(n, 1.0).expand(batch, n, n).contiguous(), _phases(n, batch, seed, rms))
    e = e.reshape(batch, n * n).to(COMPLEX[dtype])
    return e if batch > 1 else e[0].clone()


def _focal_fields(q, airy, batch, seed, dtype):
    """Speckled stellar images on a focal grid, flat."""
    u = _dev(_focal_axis(q, airy))
    m = u.numel()
    envelope = 1 / (1 + u[None, :]**2 + u[:, None]**2)
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed))
    noise = torch.randn((batch, m, m, 2), dtype=torch.float64, device=DEVICE, generator=g)
    e = envelope * torch.view_as_complex(noise)
    e = e.reshape(batch, m * m).to(COMPLEX[dtype])
    return e if batch > 1 else e[0].clone()


def _commands(case, count, seed):
    a = np.random.default_rng(seed).standard_normal((case['vectors'], count)) * 1e-3
    return _dev(a.astype(np.float32))


def _spectrum(shape, seed, dtype):
    """A field on an FFT plane: noise under the falling envelope of a turbulent pupil's spectrum."""
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed))
    noise = torch.randn(tuple(shape) + (2,), dtype=torch.float64, device=DEVICE, generator=g)
    y, x = (torch.linspace(-1, 1, s, dtype=torch.float64, device=DEVICE) for s in shape)
    return (torch.view_as_complex(noise) / (0.05 + x[None, :]**2 + y[:, None]**2)).reshape(-1).to(COMPLEX[dtype])


# ---- the framework's side ---------------------------------------------------------------------------------------


def _wavefront(field, grid, wavelength=1.0):
    return hg.Wavefront(hg.Field(field, grid), wavelength)


def _wavelengths(case):
    return [float(w) for w in np.linspace(0.9, 1.1, case['wavelengths'])]


def prepare(case, seed):
    kind = case['kind']
    n = case['n']
    s = {'kind': kind}
    if kind == 'lens':
        pupil, focal = hg.make_pupil_grid(n, 1.0), hg.make_focal_grid(case['q'], case['airy'])
        s['lens'] = hg.FraunhoferPropagator(pupil, focal, precision=case['precision'])
        s['backward'] = case['backward']
        if case['backward']:
            s['wf'] = _wavefront(_focal_fields(case['q'], case['airy'], case['batch'], seed, case['dtype']), focal)
        else:
            s['wf'] = _wavefront(_pupil_fields(n, case['batch'], seed, case['dtype']), pupil)
    elif kind == 'lyot':
        pupil, mask_grid = hg.make_pupil_grid(n, 1.0), hg.make_focal_grid(case['q'], case['airy'])
        focal = hg.make_focal_grid(case['image_q'], case['image_airy'])
        s['lyot'] = hg.LyotCoronagraph(pupil, hg.Field(_mask(case['q'], case['airy']), mask_grid),
                                       hg.Field(_disk(n, 0.9).reshape(-1), pupil), precision=case['precision'])
        s['lens'] = hg.FraunhoferPropagator(pupil, focal, precision=case['precision'])
        s['wf'] = _wavefront(_pupil_fields(n, case['batch'], seed, case['dtype'], 0.01), pupil)
    elif kind == 'gradient':
        pupil, mask_grid, focal = hg.make_pupil_grid(n, 1.0), hg.make_focal_grid(8, 32), hg.make_focal_grid(4, 32)
        pokes = hg.make_gaussian_influence_functions(pupil, case['actuators'], 1.0 / case['actuators'])
        pokes = hg.find_illuminated_actuators(pokes, _disk(n, 1.0).cpu().numpy(), 0.1)
        s['dm'] = hg.DeformableMirror(pokes)
        s['lyot'] = hg.LyotCoronagraph(pupil, hg.Field(_mask(8, 32), mask_grid),
                                       hg.Field(_disk(n, 0.9).reshape(-1), pupil), precision=case['precision'])
        s['lens'] = hg.FraunhoferPropagator(pupil, focal, precision=case['precision'])
        s['wf'] = _wavefront(_pupil_fields(n, 1, 1, 'c64', 0.01), pupil)
        s['roi'] = _dark_zone().float()
        s['commands'] = _commands(case, pokes.num_modes, seed)
    elif kind == 'vortex':
        pupil = hg.make_pupil_grid(n, 1.0)
        s['lens'] = hg.VortexCoronagraph(pupil, case['charge'])
        s['backward'] = False
        s['wf'] = _wavefront(_pupil_fields(n, 1, seed, case['dtype'], 0.05), pupil)
    elif kind == 'broadband':
        pupil, wl = hg.make_pupil_grid(n, 1.0), _wavelengths(case)
        grids = hg.diffraction_scaled_focal_grids(4, 32, wl, 1.0)
        s['field'] = _pupil_fields(n, 1, seed, 'c64')
        s['imager'] = hg.BroadbandImager(pupil, wl, grids, precision=case['precision']).capture(s['field'])
    elif kind == 'fft':
        ft = hg.FastFourierTransform(hg.make_pupil_grid(n, 1.0), case['q'], case['fov'])
        if case['backward']:
            s['ft'], s['field'] = ft.backward, hg.Field(_spectrum(ft.shape_out, seed, case['dtype']), ft.output_grid)
        else:
            s['ft'], s['field'] = ft.forward, hg.Field(_pupil_fields(n, 1, seed, case['dtype']), ft.input_grid)
    elif kind == 'asp':
        pupil = hg.make_pupil_grid(n, 8.0)
        s['lens'] = hg.AngularSpectrumPropagator(pupil, case['distance'])
        s['backward'] = case['backward']
        s['wf'] = _wavefront(_pupil_fields(n, 1, seed, case['dtype'], 2.0), pupil, 1.6e-6)
    else:
        pupil = hg.make_pupil_grid(n, 1.0)
        real = torch.float32 if case['dtype'] == 'c64' else torch.float64
        s['screen'] = _phases(n, 1, seed + 1, 2.0)[0].to(real)
        s['shift'] = _shift(seed)
        s['wf'] = _wavefront(_pupil_fields(n, 1, seed, case['dtype']), pupil)
    if kind in ('lens', 'lyot', 'gradient', 'vortex', 'asp', 'fft'):
        run(s)  # the plans of this field type, which every later pass uses
    return s


def run(s):
    kind = s['kind']
    if kind == 'lyot':
        return s['lens'].forward(s['lyot'].forward(s['wf'])).electric_field.data
    if kind == 'gradient':
        a = s['commands'].clone().requires_grad_(True)
        s['dm'].actuators = a
        image = s['lens'].forward(s['lyot'].forward(s['dm'].forward(s['wf'])))
        hg.intensity_sum(image.electric_field, s['roi']).sum().backward()
        return a.grad
    if kind == 'broadband':
        return s['imager'].replay(s['field'])
    if kind == 'fft':
        return s['ft'](s['field']).data
    if kind == 'screen':
        moved = hg.subpixel_shift(s['screen'], *s['shift'])
        return [moved, hg.PhaseApodizer(moved.reshape(-1)).forward(s['wf']).electric_field.data]
    element = s['lens']
    return (element.backward if s['backward'] else element.forward)(s['wf']).electric_field.data


# ---- what a pass cannot do without --------------------------------------------------------------------------------


def _mft_flops(n, m):
    """Two matrix products, 8 operations for each complex multiplication and addition."""
    return 8.0 * (n * n * m + m * m * n)


def _fft_flops(n):
    return 5.0 * n * n * 2 * math.log2(max(n, 2))


def work(case):
    kind, n = case['kind'], case['n']
    z = SIZE[case.get('dtype', 'c64')]
    if kind == 'lens':
        m, b = int(2 * case['q'] * case['airy']), case['batch']
        wide = 16 if case['precision'] == 'split' else z
        n_in, n_out = (m, n) if case['backward'] else (n, m)
        return {'bytes': b * (z * n_in**2 + wide * n_out**2), 'flops': b * _mft_flops(n, m)}
    if kind == 'lyot':
        m, k, b = int(2 * case['q'] * case['airy']), int(2 * case['image_q'] * case['image_airy']), case['batch']
        wide = 16 if case['precision'] == 'split' else z
        return {'bytes': b * (z * n**2 + wide * k**2) + z * (n**2 + m**2),
                'flops': b * (2 * _mft_flops(n, m) + _mft_flops(n, k))}
    if kind == 'gradient':
        count, v = 0.82 * case['actuators']**2, case['vectors']
        flops = 2 * (2 * _mft_flops(n, 512) + _mft_flops(n, 256))
        return {'bytes': v * 8 * count + 8 * n**2 + 8 * 512**2, 'flops': v * (flops + 4 * 23 * n**2)}
    if kind == 'vortex':
        return {'bytes': 2 * z * n**2, 'flops': 2 * _fft_flops(2 * n) + 5 * 2 * _mft_flops(n, 128)}
    if kind == 'broadband':
        out = [int(2 * 4 * 32 / w) for w in _wavelengths(case)]
        wide = 16 if case['precision'] == 'split' else 8
        return {'bytes': 8 * n**2 + sum(wide * m**2 for m in out), 'flops': sum(_mft_flops(n, m) for m in out)}
    if kind == 'fft':
        full = case['q'] * n
        return {'bytes': z * (n**2 + int(full * case['fov'])**2), 'flops': _fft_flops(full)}
    if kind == 'asp':
        return {'bytes': 2 * z * n**2, 'flops': 2 * _fft_flops(2 * n)}
    return {'bytes': (2 * z + z / 2 * 3) * n**2, 'flops': (2 * 14 + 20) * n**2}


# ---- the same in 64 bits --------------------------------------------------------------------------------------------


def _mask(q, airy):
    """A focal-plane mask: 0 inside an occulter of 4 lambda/D radius, flat."""
    u = _dev(_focal_axis(q, airy))
    return (u[None, :]**2 + u[:, None]**2 > 16.0).double().reshape(-1)


def _dark_zone():
    u = _dev(_focal_axis(4, 32))
    r2 = u[None, :]**2 + u[:, None]**2
    return ((r2 >= 9) & (r2 <= 144) & (u[None, :] > 0)).reshape(-1)


def _fourier(e, x, u, sign):
    """sum over x and y of e exp(sign i (u x + v y)) for square grids with the axes x and u."""
    m = torch.exp(sign * 1j * _dev(u)[:, None] * _dev(x)[None, :])
    return m @ e @ m.T


def _to_focus(e, n, q, airy, wavelength=1.0):
    return _fourier(e, _axis(n), 2 * math.pi / wavelength * _focal_axis(q, airy), -1) * (-1j / wavelength / n**2)


def _to_pupil(f, n, q, airy):
    return _fourier(f, 2 * math.pi * _focal_axis(q, airy), _axis(n), 1) * (1j / q**2)


def _coronagraph(e, n, q, airy):
    m = int(2 * q * airy)
    masked = _to_focus(e, n, q, airy) * (1 - _mask(q, airy).reshape(m, m))
    return (e - _to_pupil(masked, n, q, airy)) * _disk(n, 0.9)


def _square(e):
    n = math.isqrt(e.shape[-1])
    return e.to(torch.complex128).reshape(tuple(e.shape[:-1]) + (n, n))


def _flat(e):
    return e.reshape(tuple(e.shape[:-2]) + (-1,))


def _shift(seed):
    return tuple(float(v) for v in np.random.default_rng(seed).uniform(-0.5, 0.5, 2))


def _spline(shift):
    """The quintic B-spline at the distances of the seven nearest pixels from a point moved by `shift`."""
    t = np.arange(-3, 4) - shift
    return sum((-1)**j * math.comb(6, j) * np.maximum(t + 3 - j, 0)**5 for j in range(7)) / 120


def _moved(a, shift, dim):
    """The B-spline filter along one axis, the edge pixels repeated."""
    n = a.shape[dim]
    at = torch.arange(n, device=a.device)
    return sum(w * a.index_select(dim, (at + k - 3).clamp(0, n - 1)) for k, w in enumerate(_spline(shift)))


def _pokes(n, across):
    """Gaussian influence functions (n^2, count): crosstalk 0.15, cut off at 3 pitches, the lit actuators alone."""
    pitch, x = 1.0 / across, _dev(_axis(n))
    sigma = pitch / math.sqrt(-2 * math.log(0.15))
    reach = 3 * pitch
    disk = _disk(n, 1.0).reshape(-1)
    modes = []
    for ay in _axis(across):
        for ax in _axis(across):
            r2 = (x[None, :] - ax)**2 + (x[:, None] - ay)**2
            p = torch.exp(-0.5 * r2 / sigma**2) - math.exp(-0.5 * (reach / sigma)**2)
            p = torch.where(r2 > reach**2, torch.zeros_like(p), p).reshape(-1)
            if float((p * p * disk).sum()) >= 0.1 * float((p * p).sum()):
                modes.append(p)
    return torch.stack(modes, 1)


def _tukey(m, size):
    """A Hann window of `size` in the middle of m zeros."""
    w = np.zeros(m)
    lo = (m - size) // 2
    w[lo:lo + size] = 0.5 * (1 - np.cos(2 * np.pi * np.arange(size) / size))
    return w


def _vortex(e, n, charge):
    """The multi-scale vortex: the phase mask on nested focal grids, each level without what the coarser ones hold."""
    levels, window = 6, 32
    grids, masks = [], []
    for i in range(levels):
        q = 2 * 4**i
        m = 2 * n if i == 0 else 4 * window
        u = (np.arange(m) - m // 2) / q
        xx, yy = np.meshgrid(u, u)
        mask = np.exp(1j * charge * np.arctan2(yy, xx)) * ((xx != 0) | (yy != 0))
        if i != levels - 1:
            w = _tukey(m, window)
            mask = mask * (1 - w[:, None] * w[None, :])
        mask = _dev(mask)
        for uj, mj in zip(grids, masks):
            # the coarser mask, band-limited, at the points of this grid
            x = 2 * np.pi * (np.arange(uj.size) - uj.size // 2) / (uj.size * (uj[1] - uj[0]))
            spectrum = _fourier(mj, uj, x, -1) / uj.size**2
            mask = mask - _fourier(spectrum, x, u, 1)
        grids.append(u)
        masks.append(mask)
    # the first level filters the field padded to twice its size, the others go by dense transforms
    size = 2 * n
    padded = torch.zeros((size, size), dtype=torch.complex128, device=DEVICE)
    padded[n - n // 2:n - n // 2 + n, n - n // 2:n - n // 2 + n] = e
    out = torch.fft.ifft2(torch.fft.fft2(padded) * torch.fft.ifftshift(masks[0]))
    out = out[n - n // 2:n - n // 2 + n, n - n // 2:n - n // 2 + n].clone()
    x = _axis(n)
    for i in range(1, levels):
        k = 2 * np.pi * grids[i]
        focal = _fourier(e, x, k, -1) * masks[i] / n**2
        out += _fourier(focal, k, x, 1) * (grids[i][1] - grids[i][0])**2
    return out


def _angular_spectrum(e, n, distance, backward):
    wavelength, diameter = 1.6e-6, 8.0
    size = 2 * n
    step = 2 * math.pi / (diameter / n * size)
    k = 2 * math.pi / wavelength
    at = (np.arange(size) - size // 2) * step
    tf = 0
    for oy in (-0.25, 0.25):
        for ox in (-0.25, 0.25):
            r = np.sqrt((at + ox * step)[None, :]**2 + (at + oy * step)[:, None]**2)
            tf = tf + np.exp(1j * np.sqrt(k * k - r * r + 0j) * distance) / 4
    tf = _dev(np.fft.ifftshift(tf))
    lo = n - n // 2
    padded = torch.zeros((size, size), dtype=torch.complex128, device=DEVICE)
    padded[lo:lo + n, lo:lo + n] = e
    return torch.fft.ifft2(torch.fft.fft2(padded) * (tf.conj() if backward else tf))[lo:lo + n, lo:lo + n]


def exact(case, seed):
    kind, n = case['kind'], case['n']
    dtype = case.get('dtype', 'c64')
    if kind == 'lens':
        if case['backward']:
            f = _square(_focal_fields(case['q'], case['airy'], case['batch'], seed, dtype))
            return _flat(_to_pupil(f, n, case['q'], case['airy']))
        return _flat(_to_focus(_square(_pupil_fields(n, case['batch'], seed, dtype)), n, case['q'], case['airy']))
    if kind == 'lyot':
        e = _square(_pupil_fields(n, case['batch'], seed, dtype, 0.01))
        return _flat(_to_focus(_coronagraph(e, n, case['q'], case['airy']), n, case['image_q'], case['image_airy']))
    if kind == 'gradient':
        pokes = _pokes(n, case['actuators'])
        a = _commands(case, pokes.shape[1], seed).double()
        e0, roi, grads = _square(_pupil_fields(n, 1, 1, 'c64', 0.01)), _dark_zone().double(), []
        for part in a.split(8):
            c = part.clone().requires_grad_(True)
            e = e0 * torch.exp(4j * math.pi * (c @ pokes.T).reshape(-1, n, n))
            image = _to_focus(_coronagraph(e, n, 8, 32), n, 4, 32)
            (_flat(image.real**2 + image.imag**2) * roi).sum().backward()
            grads.append(c.grad)
        return torch.cat(grads)
    if kind == 'vortex':
        return _flat(_vortex(_square(_pupil_fields(n, 1, seed, dtype, 0.05)), n, case['charge']))
    if kind == 'broadband':
        e = _square(_pupil_fields(n, 1, seed, 'c64'))
        return [_flat(_to_focus(e, n, 4, 32.0 * 1.0 / w, w)) for w in _wavelengths(case)]
    if kind == 'fft':
        full = case['q'] * n
        m = int(n * case['fov'] * case['q'])
        k = 2 * math.pi / case['q'] * (np.arange(m) - m / 2 + (m % 2) * 0.5)
        if case['backward']:
            return _flat(_fourier(_square(_spectrum((m, m), seed, dtype)), k, _axis(n), 1) * (n / full)**2)
        return _flat(_fourier(_square(_pupil_fields(n, 1, seed, dtype)), _axis(n), k, -1) / n**2)
    if kind == 'asp':
        return _flat(_angular_spectrum(_square(_pupil_fields(n, 1, seed, dtype, 2.0)), n, case['distance'],
                                       case['backward']).contiguous())
    real = torch.float32 if dtype == 'c64' else torch.float64
    moved = _moved(_moved(_phases(n, 1, seed + 1, 2.0)[0].to(real).double(), _shift(seed)[1], 1), _shift(seed)[0], 0)
    return [moved, _flat(_square(_pupil_fields(n, 1, seed, dtype)) * torch.exp(1j * moved))]
