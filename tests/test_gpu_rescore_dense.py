"""The dense frames' rescoring (rspi_rescore_dense) against the sparse
entries' (rspi_rescore) on the same candidates: the same FP64 terms in
another order, each sum within n 2^-53 of its terms' magnitudes (n below
1e4, the terms' sum below 1e2 of the largest likelihood here)."""
import numpy as np
import pytest
import torch

from helpers import random_photons
from oracle import emc_oracle as E

pytestmark = pytest.mark.gpu


# one partial tile of 2,048 columns, exactly over one, three; few candidates
# (the argmax alone), and every state of every frame (chunks across rows)
@pytest.mark.parametrize('size', [25, 54, 85])
@pytest.mark.parametrize('delta', [0., 1e9])
def test_dense_rescoring_equals_sparse(size, delta):
    from rspi.device import DevicePhotons, EStep, cur_stream, ptr
    from rspi.lib import call
    n, num_rot = 37, 5
    d = random_photons(size, n, 3. * size * size, size, empty_frames=(1,))
    ds = E.parse_photons(d['ones'], d['multi'], d['place_ones'], d['place_multi'],
                         d['count_multi'], size * size, True)
    frames = np.asarray(E.sparse_frames(ds).todense()).astype(np.uint16)
    ph = DevicePhotons(d['ones'], d['multi'], d['place_ones'], d['place_multi'],
                       d['count_multi'], size * size, True, frames=frames)
    sx, sy, dia, _ = E.generate_states((-1., 1., 2), (0., 1., 2), (6., 8., 2))
    _, pm = E.generate_masks(size)
    es = EStep(ph, size, num_rot, sx, sy, dia, pm, ds['bg'], form='dense', delta=delta)
    rng = np.random.default_rng(size)
    es.run(torch.from_numpy(rng.random(size * size) + 1j * rng.random(size * size)).cuda())
    es.reduce()
    total = es.n_candidates
    assert total == (es.n_rows * n if delta else total) and total >= n
    got = es.cand_ll[:total].clone()
    call('rspi_rescore', ptr(es.cand_d), ptr(es.cand_r), ptr(es.cand_off), n, es.capacity,
         es.n_rows, ptr(es.holo), num_rot, ptr(es.rot_cs), size, ptr(es.bg), ptr(es.sel_pix),
         es.n_sel, es.p_pad, ptr(es.init), ptr(ph.scales), ptr(es.ll['entries']),
         ptr(es.ll['row_off']), ptr(es.row_cnt), ptr(es.row_cand_off), ptr(es.row_cand),
         ptr(es.cand_ll), ptr(es.prob), ptr(es.max32), ptr(es.noncand), ptr(es.maxll),
         ptr(es.rmax), ptr(es.logz), ptr(es.row_scratch), es.scratch_rows, cur_stream())
    want = es.cand_ll[:total]
    ph.err.check('rescore')
    assert float((got - want).abs().max()) <= 1e-10 * float(want.abs().max())
