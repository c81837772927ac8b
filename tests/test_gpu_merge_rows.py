"""The row-grouped merge (rspi_merge_rows) against the pair-by-pair one
(rspi_merge) on the same candidates: rows with enough photons to be summed
unrotated first, rows without, and rows without a pair.  Both add the same
positive FP64 terms in other orders (at most 1e6 of them: 1e6 2^-53)."""
import numpy as np
import pytest
import torch

from helpers import random_photons
from oracle import emc_oracle as E

pytestmark = pytest.mark.gpu


# photons per frame from a few to several per pixel; odd and even detectors;
# fewer images than rows (a CTA takes several) and one image only
@pytest.mark.parametrize('size,n,photons', [(21, 12, 30.), (21, 40, 400.), (36, 60, 2000.)])
@pytest.mark.parametrize('images', [1, 7, 296])
def test_merge_rows_equals_pairs(size, n, photons, images):
    from rspi.device import DevicePhotons, EStep, Merge, cur_stream, ptr
    from rspi.lib import call
    num_rot = 6
    d = random_photons(size, n, photons, size + n, empty_frames=(1,))
    ds = E.parse_photons(d['ones'], d['multi'], d['place_ones'], d['place_multi'],
                         d['count_multi'], size * size, True)
    ph = DevicePhotons(d['ones'], d['multi'], d['place_ones'], d['place_multi'],
                       d['count_multi'], size * size, True)
    sx, sy, dia, _ = E.generate_states((-1., 1., 2), (0., 1., 2), (4., 6., 2))
    _, pm = E.generate_masks(size)
    es = EStep(ph, size, num_rot, sx, sy, dia, pm, ds['bg'], form='screen', delta=20.)
    rng = np.random.default_rng(size)
    es.run(torch.from_numpy(rng.random(size * size) + 1j * rng.random(size * size)).cuda())
    es.reduce()
    mg = Merge(es)
    mg.images = mg.images[:images]
    got = mg.run().clone()
    got_w = mg.w.clone()
    call('rspi_merge', ptr(es.cand_d), ptr(es.cand_r), ptr(es.cand_ll), ptr(es.cand_off[n:]),
         es.capacity, ptr(es.logz), mg.p_min, ptr(ph.scales), ptr(ph.ones), ptr(ph.multi),
         ptr(ph.ones_accum), ptr(ph.multi_accum), ptr(ph.place_ones), ptr(ph.place_multi),
         ptr(ph.count_multi), es.n_states0, num_rot, ptr(es.rot_cs), size, ptr(mg.cov),
         ptr(mg.num), ptr(mg.den), ptr(mg.w), ptr(mg.intens), cur_stream())
    ph.err.check('merge')
    np.testing.assert_allclose(got_w.cpu().numpy(), mg.w.cpu().numpy(), rtol=1e-10)
    np.testing.assert_allclose(got.cpu().numpy(), mg.intens.cpu().numpy(), rtol=1e-9, atol=1e-300)
