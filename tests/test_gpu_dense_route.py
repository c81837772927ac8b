"""Which kernel rescores the dense form's candidates: over all columns where
the photons fill most of them, else over the entries, whose cost is that of
the photons."""
import numpy as np
import pytest
import torch

from oracle import emc_oracle as E

pytestmark = pytest.mark.gpu


# size 41: the FP64 row fits shared memory; 215 (36,000 columns): it does not
@pytest.mark.parametrize('size,mean,columns', [
    (41, 0.05, False), (41, 0.6, False), (41, 2.5, True),
    (215, 0.05, False), (215, 0.3, False), (215, 0.7, True)])
def test_rescoring_route(size, mean, columns, monkeypatch):
    """Poisson counts of `mean` per pixel fill 1 - exp(-mean) of the columns."""
    from rspi import device
    from rspi.photonfile import sparse_from_dense
    n, num_rot = 9, 3
    rng = np.random.default_rng(size)
    frames = rng.poisson(mean, (n, size * size)).astype(np.uint16)
    d = sparse_from_dense(frames)
    ds = E.parse_photons(d['ones'], d['multi'], d['place_ones'], d['place_multi'],
                         d['count_multi'], size * size, True)
    ph = device.DevicePhotons(d['ones'], d['multi'], d['place_ones'], d['place_multi'],
                              d['count_multi'], size * size, True, frames=frames)
    sx, sy, dia, _ = E.generate_states((0., 1., 2), (0., 0., 1), (6., 8., 2))
    _, pm = E.generate_masks(size)
    es = device.EStep(ph, size, num_rot, sx, sy, dia, pm, ds['bg'], form='dense')
    seen = []
    call = device.call
    monkeypatch.setattr(device, 'call', lambda name, *a: (seen.append(name), call(name, *a))[1])
    model = rng.random(size * size) + 1j * rng.random(size * size)
    es.run(torch.from_numpy(model).cuda())
    maxll, rmax, logz = es.reduce()
    assert ('rspi_rescore_dense' in seen) == columns
    assert ('rspi_rescore' in seen) == (not columns)
    want, _, _ = E.calc_prob(model, ds, sx, sy, dia, size, num_rot, pm, E.get_scales(ds, True))
    mx, am = E.get_rmax(want)
    assert np.array_equal(rmax.cpu().numpy(), am)
    np.testing.assert_allclose(maxll.cpu().numpy(), mx, rtol=1e-11)
    np.testing.assert_allclose(logz.cpu().numpy(), E.posterior(want)[0], rtol=1e-11)
