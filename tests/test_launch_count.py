"""Launches counted per call: those of a call's scan depend on its length
(counted here with the entry points replaced: no GPU)."""
import re

import pytest

from conftest import REPO
from rspi import lib as rlib


def arguments(name):
    text = open(REPO + '/include/rspi.h').read()
    return re.search(r'\b%s\s*\(([^;]*)\);' % name, text, re.S).group(1).split(',')


# up to 4 tiles of 4,096 counts one launch, beyond three
@pytest.mark.parametrize('n,scan', [(1, 1), (16384, 1), (16385, 3), (10 ** 7, 3)])
@pytest.mark.parametrize('name,length,kernels', [
    ('rspi_scan_rows', 'n_data', 0), ('rspi_screen_candidates', 'n_data', 2),
    ('rspi_screen_candidates_cols', 'n_data', 3), ('rspi_screen_candidates_noalloc', 'n_data', 2),
    ('rspi_rescore', 'n_rows', 4), ('rspi_rescore_cols', 'n_rows', 4),
    ('rspi_rescore_dense', 'n_rows', 3), ('rspi_posterior_pairs', 'n_data', 2),
    ('rspi_maxlp_pixel_map', 'num_rot', 2)])
def test_scan_launches_are_counted(name, length, kernels, n, scan, monkeypatch):
    args = [0] * len(arguments(name))
    for i, a in enumerate(arguments(name)):
        if a.split()[-1] == length:
            args[i] = n
        elif a.split()[-1] == 'size':
            args[i] = 1

    class Fake:
        rspi_scan_launches = staticmethod(rlib.load().rspi_scan_launches)

        def __getattr__(self, _):
            return lambda *a: 0

    monkeypatch.setattr(rlib, '_lib', Fake())
    before = rlib.launch_count
    rlib.call(name, *args)
    assert rlib.launch_count - before == kernels + scan
