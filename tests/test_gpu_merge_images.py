"""The merge's unrotated images stay within the rows there are and a byte
budget, whatever the detector; the intensities do not depend on their
number."""
import numpy as np
import pytest
import torch

from helpers import random_photons
from oracle import emc_oracle as E
from rspi import device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('size,num_rot', [(21, 6), (36, 40)])
def test_images_within_rows_and_budget(size, num_rot, monkeypatch):
    n, npix = 40, size * size
    d = random_photons(size, n, float(npix), size, empty_frames=(1,))
    ds = E.parse_photons(d['ones'], d['multi'], d['place_ones'], d['place_multi'],
                         d['count_multi'], npix, True)
    ph = device.DevicePhotons(d['ones'], d['multi'], d['place_ones'], d['place_multi'],
                              d['count_multi'], npix, True)
    sx, sy, dia, _ = E.generate_states((-1., 1., 2), (0., 1., 2), (4., 6., 2))
    _, pm = E.generate_masks(size)
    es = device.EStep(ph, size, num_rot, sx, sy, dia, pm, ds['bg'], form='screen', delta=20.)
    rng = np.random.default_rng(size)
    es.run(torch.from_numpy(rng.random(npix) + 1j * rng.random(npix)).cuda())
    es.reduce()
    want = device.Merge(es)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert want.images.shape[0] == min(2 * sms, es.n_rows)
    want = want.run().cpu().numpy()
    for images in (5, 0):                      # 0: one image is the least
        monkeypatch.setattr(device, 'MERGE_IMAGES', images * 8 * npix + 7)
        mg = device.Merge(es)
        assert mg.images.shape[0] == max(1, images)
        # positive FP64 terms in another order, at most 1e6 of them
        np.testing.assert_allclose(mg.run().cpu().numpy(), want, rtol=1e-9, atol=1e-300)
    ph.err.check('merge')
