"""FP32 form of the grid NLLs: every pixel's gradient term is widened to FP64
before terms are added.  Two large terms that cancel exactly must not take
the small ones of their opposite or quarter-turned pixels with them."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

BIG = 1.5 * 2. ** 34    # 2,048 between FP32 neighbours: 1,000 beside it is lost
SMALL = 1000.           # the reference amplitude (< 1/3) beside it: 3.4e-4


@pytest.mark.parametrize('kind', ['pixel', 'slicing'])
def test_opposite_terms_are_widened_first(kind):
    from rspi import adjoint, geometry
    from rspi.device import DevicePhotons
    size, c = 41, 20
    # photons in two corners of the detector, which no mask keeps: the dense part alone
    i = lambda *v: np.array(v, 'i4')  # noqa: E731
    ph = DevicePhotons(i(1), i(1), i(0), i(size - 1), i(2), size * size)
    if kind == 'pixel':
        prob = adjoint.NLLProblem(ph, size, [0.3], precision='fp32')
        at = {int(p): i for i, p in enumerate(prob.pixels)}
        n = prob.n_pix
    else:
        mask = geometry.emc_masks(size)[1]
        prob = adjoint.EMCNLLProblem(ph, size, np.array([[1., 0.]]), mask,
                                     np.zeros(size * size), 1., precision='fp32')
        at = {int(p): int(p) for p in np.flatnonzero(np.asarray(mask).ravel() == 0)}
        n = size * size
    assert prob._grid is not None
    place = lambda x, y: at[(x + c) * size + y + c]  # noqa: E731
    t = lambda a: torch.from_numpy(np.asarray(a, dtype='f8')).cuda()  # noqa: E731
    one = lambda v: t([v])  # noqa: E731
    # no shift: e^{i th} = 1 and all pixels of radius 10 share ff and dff / ddia
    par = (one(5.), one(0.), one(0.), one(1.))
    # diameter: Re F of two orbits, BIG and -BIG, their opposites SMALL
    re = np.zeros(n)
    re[place(8, 6)], re[place(-8, -6)] = BIG, SMALL
    re[place(6, 8)], re[place(-6, -8)] = -BIG, SMALL
    # shift x: Im F; (8, 6) and (-8, 6) have opposite x, their opposites SMALL
    im = np.zeros(n)
    im[place(8, 6)], im[place(-8, 6)] = BIG, BIG
    im[place(-8, -6)], im[place(8, -6)] = -SMALL, SMALL
    zero = np.zeros(n)
    for parts, which in (((re, zero), 2), ((zero, im), 3)):
        base = prob.evaluate(t(zero), t(zero), *par, grad=True)[1][which]
        got = prob.evaluate(t(parts[0]), t(parts[1]), *par, grad=True)[1][which] - base
        grid, prob._grid = prob._grid, None
        want = prob.evaluate(t(parts[0]), t(parts[1]), *par, grad=True)[1][which] - base
        prob._grid = grid
        # the reference amplitudes lost beside BIG: 2 x 3.4e-4 of SMALL
        assert float(want.abs()) > 0.
        assert float((got - want).abs()) <= 2e-3 * float(want.abs())
