"""The dense sums of the two differentiable likelihoods from the detector
grid's tables (rspi_nll_grid, rspi_emc_nll_grid) against the general kernels
(rspi_nll, rspi_emc_nll), in FP64: both sum the same terms in FP64, each
within a few roundings (2^-53) of its value, over at most 1e6 terms."""
import numpy as np
import pytest
import torch

from helpers import random_photons

pytestmark = pytest.mark.gpu


# frames: one, around the four of a round, more than one block of frames;
# sizes: two orbits, odd and even, more than one group of orbits (256 in FP64)
@pytest.mark.parametrize('size,n', [(11, 1), (11, 3), (18, 4), (18, 5), (41, 33), (50, 257)])
@pytest.mark.parametrize('kind', ['pixel', 'slicing'])
def test_grid_tables_equal_general(size, n, kind):
    from rspi import adjoint, geometry
    from rspi.device import DevicePhotons
    d = random_photons(size, n, 4. * size, 3 * size + n)
    ph = DevicePhotons(d['ones'], d['multi'], d['place_ones'], d['place_multi'],
                       d['count_multi'], size * size)
    rng = np.random.default_rng(size + n)
    ang = rng.uniform(0., 2 * np.pi, n)
    if kind == 'pixel':
        prob = adjoint.NLLProblem(ph, size, ang, precision='fp64')
        npix = prob.n_pix
    else:
        cs = np.stack([np.cos(ang), np.sin(ang)], 1)
        prob = adjoint.EMCNLLProblem(ph, size, cs, geometry.emc_masks(size)[1],
                                     rng.uniform(0., 0.3, size * size), 0.7, precision='fp64')
        npix = size * size
    t = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    args = (t(rng.standard_normal(npix)), t(rng.standard_normal(npix)), t(rng.uniform(4., 8., n)),
            t(rng.uniform(-3., 3., n)), t(rng.uniform(-3., 3., n)), t(rng.uniform(0.5, 2., n)))
    assert prob._grid is not None
    got, g = prob.evaluate(*args, grad=True)
    got0 = prob.evaluate(*args)
    prob._grid = None
    want, w = prob.evaluate(*args, grad=True)
    ph.err.check('nll')
    assert abs(float(got - want)) <= 1e-12 * abs(float(want))
    assert abs(float(got0 - want)) <= 1e-12 * abs(float(want))
    for a, b in zip(g, w):
        tol = 1e-11 * float(b.abs().max())
        assert float((a - b).abs().max()) <= tol


def test_value_and_gradient_modes():
    """Under no_grad, and for inputs that need no gradient, the value pass
    gives the gradient pass's value; a second backward gives the same."""
    from rspi import adjoint
    from rspi.device import DevicePhotons
    size, n = 21, 6
    d = random_photons(size, n, 100., 4)
    ph = DevicePhotons(d['ones'], d['multi'], d['place_ones'], d['place_multi'],
                       d['count_multi'], size * size)
    rng = np.random.default_rng(1)
    prob = adjoint.NLLProblem(ph, size, rng.uniform(0., 6., n), precision='fp64')
    t = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    args = [t(rng.standard_normal(prob.n_pix)), t(rng.standard_normal(prob.n_pix)),
            t(rng.uniform(4., 8., n)), t(rng.uniform(-1., 1., n)), t(rng.uniform(-1., 1., n)),
            t(rng.uniform(0.5, 2., n))]
    plain = adjoint.nll(prob, *args)
    assert not plain.requires_grad
    args[0].requires_grad_(True)
    loss = adjoint.nll(prob, *args)
    with torch.no_grad():
        quiet = adjoint.nll(prob, *args)
    assert not quiet.requires_grad and loss.requires_grad
    for v in (loss, quiet):
        assert abs(float(v.detach() - plain)) <= 1e-12 * abs(float(plain))
    g1, = torch.autograd.grad(loss, args[0], retain_graph=True)
    g2, = torch.autograd.grad(2. * loss, args[0])
    assert torch.equal(2. * g1, g2)
