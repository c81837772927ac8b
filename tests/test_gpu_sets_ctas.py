"""Changing the frame-set kernel's CTA count after construction: one column
part has no scratch that depends on it, so the entries stay, also under
capture; the likelihoods do not depend on it."""
import numpy as np
import pytest
import torch

from rspi import device
from test_sets_items import _data

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('shares', [0, 10 ** 9])     # every set cut, none
@pytest.mark.parametrize('n_ctas', [1, 37, 300])
def test_entries_stay(n_ctas, shares, monkeypatch):
    from test_gpu_estep import _estep, _photons
    monkeypatch.setattr(device, 'SPLIT_SHARES', shares)
    size, ds, (sx, sy, dia, _) = _data(61, 40.)
    rng = np.random.default_rng(5)
    model = torch.from_numpy(rng.random(size * size) + 1j * rng.random(size * size)).cuda()
    es = _estep(_photons(ds, False), size, 5, sx, sy, dia, ds['bg'], form='screen',
                states_per_tile=4)
    assert es.wide['n_parts'] == 1 and (es.wide['seg_slots'] > 0) == (shares == 0)
    es.run(model)
    want = es.frame_prob().clone()   # not the last set's columns without a frame
    entries = es.wide['entries']
    es.n_ctas = n_ctas
    es.prob.zero_()
    es.run(model)
    assert es.wide['entries'] is entries
    assert torch.equal(es.frame_prob(), want)
    es.n_ctas = n_ctas + 1
    es.prob.zero_()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        es.run(model)
    graph.replay()
    torch.cuda.synchronize()
    assert es.wide['entries'] is entries
    assert torch.equal(es.frame_prob(), want)
    es.ph.err.check('frame-set kernel')
