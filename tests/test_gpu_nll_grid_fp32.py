"""The dense part of the grid NLLs in FP32 (two orbits per thread, 512 per
group) against plain torch in FP64: part of the second orbits filled, one
group and several.  The photons lie in two corners that no mask keeps.

A term's FP32 value is off by at most 16 roundings (2^-20) of its parts:
amplitudes (sin s - s cos s) / s^3 and their derivative cancel, so their
parts' magnitudes count, and |z| <= |F| + |r|.  All sums are FP64."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('size,n', [(41, 1), (41, 37), (64, 5), (101, 3), (101, 130)])
@pytest.mark.parametrize('kind', ['pixel', 'slicing'])
def test_fp32_grid_terms(size, n, kind):
    from rspi import adjoint, geometry
    from rspi.device import DevicePhotons
    rng = np.random.default_rng(size + n)
    one = np.ones(n, 'i4')
    ph = DevicePhotons(one, one, 0 * one, (size - 1) * one, 2 * one, size * size)
    ang = rng.uniform(0., 2. * np.pi, n)
    if kind == 'pixel':
        prob = adjoint.NLLProblem(ph, size, ang, precision='fp32')
        at = torch.arange(prob.n_pix, device='cuda')
        qx, qy, vscale, bg, n_model = prob.qx, prob.qy, 1., 0., prob.n_pix
    else:
        levels = rng.uniform(0., 0.3, size * size)
        prob = adjoint.EMCNLLProblem(ph, size, np.stack([np.cos(ang), np.sin(ang)], 1),
                                     geometry.emc_masks(size)[1], levels, 0.7, precision='fp32')
        at = prob.sel_pix.long()
        qx = (at // size - size // 2).double() / size
        qy = (at % size - size // 2).double() / size
        vscale, bg, n_model = 0.7, float(levels[at.cpu().numpy()].sum()), size * size
    assert prob._grid is not None
    orbits = at.numel() // 4
    assert (256 < orbits < 512) if size == 41 else orbits > 512
    t = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    re, im = t(rng.standard_normal(n_model)), t(rng.standard_normal(n_model))
    par = [t(rng.uniform(4., 8., n)), t(rng.uniform(-3., 3., n)), t(rng.uniform(-3., 3., n)),
           t(rng.uniform(0.5, 2., n))]
    got, g = prob.evaluate(re, im, *par, grad=True)
    got0 = prob.evaluate(re, im, *par)

    dia, sx, sy, scale = (v[:, None] for v in par)
    k = np.pi * torch.sqrt(qx * qx + qy * qy)[None]
    s = k * dia
    ff = (torch.sin(s) - s * torch.cos(s)) / s ** 3
    dff = (torch.sin(s) / s ** 2 - 3. * ff / s) * k
    e = torch.exp(2j * np.pi * (qx * sx + qy * sy))
    z = (re + 1j * im)[at][None] + ff * e
    parts = (1. + s) / s ** 3                              # of ff
    dparts = (1. / s ** 2 + 3. * parts / s) * k            # of dff / ddia
    zabs = (re + 1j * im)[at].abs()[None] + parts
    v = vscale * scale
    eps = 2. ** -20

    def near(a, want, magnitude):
        assert bool(((a - want).abs() <= eps * magnitude).all())

    value, size_v = (v * z.abs() ** 2).sum() + bg * v.sum(), (v * zabs ** 2).sum() + bg * v.sum()
    near(got, value, size_v)
    near(got0, value, size_v)
    near(g[0][at], 2. * (v * z.real).sum(0), 2. * (v * zabs).sum(0))
    near(g[1][at], 2. * (v * z.imag).sum(0), 2. * (v * zabs).sum(0))
    near(g[2], 2. * (v * dff * (z.conj() * e).real).sum(1), 2. * (v * dparts * zabs).sum(1))
    turn = (z.conj() * 1j * ff * e).real * 4. * np.pi * v
    for i, q in ((3, qx), (4, qy)):
        near(g[i], (q * turn).sum(1), 4. * np.pi * (v * q.abs() * parts * zabs).sum(1))
    near(g[5], vscale * ((z.abs() ** 2).sum(1) + bg), vscale * ((zabs ** 2).sum(1) + bg))
