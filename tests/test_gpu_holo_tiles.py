"""Holographic slices and their masked sums at the edges of the tiles (1,024
pixels) and of the sums' unrolled rounds (2,048 likelihood pixels), against
the FP64 oracle: each value within a few roundings, each sum within n 2^-53
(n < 1e4 positive terms)."""
import numpy as np
import pytest
import torch

from oracle import emc_oracle as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('size', [5, 32, 33, 51, 64, 101])
@pytest.mark.parametrize('n_states', [1, 3])
def test_holo_slices(size, n_states):
    from rspi.device import cur_stream, ptr
    from rspi.lib import call
    rng = np.random.default_rng(size)
    npix = size * size
    model = rng.standard_normal(npix) + 1j * rng.standard_normal(npix)
    sx, sy = rng.uniform(-3., 3., (2, n_states))
    dia, bg = rng.uniform(6., 8., n_states), rng.uniform(0., 1., npix)
    _, pm = E.generate_masks(size)
    sel = np.flatnonzero(pm < 1).astype('i4')
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    d = [t(a) for a in (model, sx, sy, dia, bg, sel if sel.size else np.zeros(1, 'i4'))]
    holo = torch.full((n_states, npix), np.nan, dtype=torch.float64, device='cuda')
    msum = torch.full((n_states,), np.nan, dtype=torch.float64, device='cuda')
    call('rspi_holo_slices', ptr(d[0]), ptr(d[1]), ptr(d[2]), ptr(d[3]), n_states, size, ptr(d[4]),
         ptr(d[5]), sel.size, ptr(holo), ptr(msum), cur_stream())
    for s in range(n_states):
        want = E.holo_slice(model, sx[s], sy[s], dia[s], 1., 1., size, bg)
        np.testing.assert_allclose(holo[s].cpu().numpy(), want, rtol=1e-11)
        np.testing.assert_allclose(float(msum[s]), want[sel].sum(), rtol=1e-11)
