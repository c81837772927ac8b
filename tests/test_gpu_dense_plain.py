"""The dense form beyond the paired slices' byte budget: digits from the plain
slices, the same likelihoods to the bit."""
import numpy as np
import pytest
import torch

from oracle import emc_oracle as E
from rspi import device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('fits', [True, False])
def test_dense_form_at_the_pairs_budget(fits, monkeypatch):
    from rspi.photonfile import sparse_from_dense
    size, n, num_rot = 37, 21, 5
    rng = np.random.default_rng(3)
    frames = rng.poisson(2., (n, size * size)).astype(np.uint16)
    d = sparse_from_dense(frames)
    ds = E.parse_photons(d['ones'], d['multi'], d['place_ones'], d['place_multi'],
                         d['count_multi'], size * size, True)
    ph = device.DevicePhotons(d['ones'], d['multi'], d['place_ones'], d['place_multi'],
                              d['count_multi'], size * size, True, frames=frames)
    sx, sy, dia, _ = E.generate_states((-1., 1., 3), (0., 0., 1), (6., 8., 2))
    _, pm = E.generate_masks(size)
    model = torch.from_numpy(rng.random(size * size) + 1j * rng.random(size * size)).cuda()

    def run():
        es = device.EStep(ph, size, num_rot, sx, sy, dia, pm, ds['bg'], form='dense')
        es.run(model)
        return es, [t.clone() for t in es.reduce()], es.prob.clone()

    _, want, prob = run()
    need = len(sx) * size * size * 16
    monkeypatch.setattr(device, 'DENSE_PAIRS', need if fits else need - 1)
    es, got, got_prob = run()
    assert es.dense_gemm == 'i8' and (es.holo_pairs is not None) == fits
    assert torch.equal(got_prob, prob)
    assert all(torch.equal(a, b) for a, b in zip(got, want))
