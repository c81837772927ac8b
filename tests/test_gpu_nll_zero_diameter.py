"""Frames whose sphere has diameter 0 in the slicing likelihood: the grid's
tables (rspi_emc_nll_grid) take the form factor of s = 1e-5 there with no
derivative, as the slices and rspi_emc_nll do."""
import numpy as np
import pytest
import torch

from helpers import random_photons

pytestmark = pytest.mark.gpu


# FP64: (sin s - s cos s) / s^3 at s = 1e-5 cancels to within 3 roundings of
# 1e-5, 3.4e-6 of a form factor of 1/3, and |M| is of order 1.  FP32: phases
# and arguments up to 30, rounded at 2^-24 in each term of rspi_emc_nll; the
# form factor cancels to 0 in both.
@pytest.mark.parametrize('precision,tol', [('fp64', 1e-5), ('fp32', 1e-4)])
@pytest.mark.parametrize('dia', [[0.], [7., 0., 6., 0., 0.], [0., 6.5, 7., 6., 8., 7.]])
def test_zero_diameter(dia, precision, tol):
    from rspi import adjoint, geometry
    from rspi.device import DevicePhotons
    size, n = 41, len(dia)
    d = random_photons(size, n, 4. * size, n)
    ph = DevicePhotons(d['ones'], d['multi'], d['place_ones'], d['place_multi'],
                       d['count_multi'], size * size)
    rng = np.random.default_rng(n)
    ang = rng.uniform(0., 2 * np.pi, n)
    prob = adjoint.EMCNLLProblem(ph, size, np.stack([np.cos(ang), np.sin(ang)], 1),
                                 geometry.emc_masks(size)[1], rng.uniform(0., 0.3, size * size),
                                 0.7, precision=precision)
    t = lambda a: torch.from_numpy(np.asarray(a)).cuda()  # noqa: E731
    args = (t(rng.standard_normal(size * size)), t(rng.standard_normal(size * size)), t(dia),
            t(rng.uniform(-3., 3., n)), t(rng.uniform(-3., 3., n)), t(rng.uniform(0.5, 2., n)))
    assert prob._grid is not None
    got, g = prob.evaluate(*args, grad=True)
    got0 = prob.evaluate(*args)
    prob._grid = None
    want, w = prob.evaluate(*args, grad=True)
    ph.err.check('nll')
    assert np.isfinite(float(want))
    assert abs(float(got - want)) <= tol * abs(float(want))
    assert abs(float(got0 - want)) <= tol * abs(float(want))
    for a, b in zip(g, w):
        assert float((a - b).abs().max()) <= tol * max(float(b.abs().max()), 1.)
