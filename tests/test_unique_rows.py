"""The phaser's grouping of per-frame (shift, diameter) rows against
np.unique, on the CPU: repeated and single rows, both zeros, one frame."""
import numpy as np
import pytest


@pytest.mark.parametrize('n', [1, 2, 7, 1000])
def test_unique_rows(n):
    maxlp = pytest.importorskip('maxLP')
    rng = np.random.default_rng(n)
    rows = np.stack([rng.choice([-1.5, -0., 0., 2.], n), rng.integers(-2, 3, n) * 0.5,
                     rng.choice([6., 6. + 1e-15, 8.], n)], axis=1)
    ref, place = maxlp._unique_rows(rows)
    want, inv = np.unique(rows, axis=0, return_inverse=True)
    assert np.array_equal(ref, want) and np.array_equal(place, inv.ravel())
    assert np.array_equal(ref[place], rows)
