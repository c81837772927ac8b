"""The screened pattern search's cells, expansion and set-up at their edges:
bit-identical to the plain FP64 search."""
import numpy as np
import pytest

from test_gpu_pattern_screen import _check_same, _random_case, _run_both

pytestmark = pytest.mark.gpu


# one reference state (a pixel's candidates tie around a circle), a round of
# 128 states and its neighbours, the most the shared memory holds; model
# values around the reference's and far below it (the expansion's regime)
@pytest.mark.parametrize('n_states', [1, 2, 127, 128, 129, 1024])
@pytest.mark.parametrize('level', [1., 1e-4, 1e-9])
def test_screened_search_edges(n_states, level, tmp_path):
    size, n = 18, 1500
    path, params, rng = _random_case(tmp_path, size, n, n_states, 100 + n_states)
    model = level * (rng.random(size * size) + 1j * rng.random(size * size))
    st = _check_same(_run_both(path, size, params, model))
    assert st[0] > 0


def test_screened_search_few_frames(tmp_path):
    """Pixels with no photon, one photon, and ring pixels without any."""
    size = 25
    path, params, rng = _random_case(tmp_path, size, 9, 4, 3, mean_factor=2.)
    model = rng.random(size * size) + 1j * rng.random(size * size)
    _check_same(_run_both(path, size, params, model))
