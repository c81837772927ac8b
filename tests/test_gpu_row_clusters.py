"""The passes over a likelihood matrix whose rows a cluster of CTAs shares
(from 1,024 rows on, for few frames): per-frame reduction and candidate
selection, against NumPy.  Rows around the points where the clusters grow;
ties, NaN and the float range's lowest value among the entries."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

ROWS = [1, 31, 33, 1023, 1024, 1025, 2049, 4096 + 37, 9001]


def _matrix(n_rows, n, seed, dtype):
    rng = np.random.default_rng(seed)
    ll = np.round(rng.normal(-50., 15., (n_rows, n)), 1).astype(dtype)   # ties
    ll[rng.random((n_rows, n)) < 0.01] = np.finfo('f4').min
    return ll


@pytest.mark.parametrize('n_rows', ROWS)
@pytest.mark.parametrize('n', [1, 33])
def test_frame_reduce(n_rows, n):
    from rspi.device import cur_stream, ptr
    from rspi.lib import call
    ll = _matrix(n_rows, n, n_rows + n, 'f8')
    if n > 2 and n_rows > 3:
        ll[n_rows - 2, 2] = np.nan
    d = torch.from_numpy(ll).cuda()
    mx = torch.empty(n, dtype=torch.float64, device='cuda')
    am = torch.empty(n, dtype=torch.int32, device='cuda')
    lz = torch.empty(n, dtype=torch.float64, device='cuda')
    call('rspi_frame_reduce', ptr(d), 1, n_rows, n, ptr(mx), ptr(am), ptr(lz), cur_stream())
    assert np.array_equal(am.cpu().numpy(), ll.argmax(0))
    assert np.array_equal(mx.cpu().numpy(), ll.max(0), equal_nan=True)
    ok = ~np.isnan(ll).any(0)
    want = ll.max(0) + np.log(np.exp(ll - ll.max(0)).sum(0))
    # n_rows additions of positive FP64 terms
    np.testing.assert_allclose(lz.cpu().numpy()[ok], want[ok], rtol=1e-11)


@pytest.mark.parametrize('n_rows', ROWS)
@pytest.mark.parametrize('delta', [0., 12., 1e6])
@pytest.mark.parametrize('cols', [False, True])
def test_candidates(n_rows, delta, cols):
    from rspi.device import cur_stream, ptr
    from rspi.lib import call
    n = 37
    ll = _matrix(n_rows, n, n_rows, 'f4')
    frame = np.random.default_rng(1).permutation(n).astype('i4') if cols else np.arange(n)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    z = lambda dt, *s: torch.zeros(s, dtype=dt, device='cuda')  # noqa: E731
    order = np.argsort(frame)                       # column of each frame
    mx, am = ll.max(0)[order].astype('f8'), ll.argmax(0)[order].astype('i4')
    cap = n_rows * n
    d_ll, d_mx, d_am, d_fr = t(ll), t(mx), t(am), t(frame.astype('i4'))
    phot, rows, lmax = z(torch.int64, n), z(torch.int64, n + 1), z(torch.float32, 1)
    cnt, slot, cn = z(torch.int32, n * 32), z(torch.int32, n * 32), z(torch.int32, n)
    nc, thr, off = z(torch.float64, n), z(torch.float64, n), z(torch.int64, n + 1)
    cd, cr, err = z(torch.int32, cap), z(torch.int32, cap), z(torch.int32, 1)
    tail = (ptr(d_am), ptr(phot), ptr(rows), ptr(lmax), delta, ptr(cnt), ptr(cn), ptr(nc),
            ptr(thr), ptr(off), cap, ptr(cd), ptr(cr))
    if cols:
        call('rspi_screen_candidates_cols', ptr(d_ll), n_rows, n, ptr(d_fr), n, ptr(d_mx), *tail,
             ptr(slot), ptr(err), cur_stream())
    else:
        call('rspi_screen_candidates', ptr(d_ll), n_rows, n, ptr(d_mx), *tail, ptr(err),
             cur_stream())
    assert int(err.item()) == 0
    off, cd, cr = off.cpu().numpy(), cd.cpu().numpy(), cr.cpu().numpy()
    for d in range(n):
        v = ll[:, order[d]].astype('f8')
        keep = (v >= float(thr[d])) | (np.arange(n_rows) == am[d])
        want = sorted(np.flatnonzero(keep), key=lambda r: (r % 32, r))
        assert np.array_equal(cr[off[d]:off[d + 1]], want)
        assert np.all(cd[off[d]:off[d + 1]] == d)
        # FP32 exponentials (2 ulps each), summed in FP64
        np.testing.assert_allclose(float(nc[d]), np.exp(v[~keep] - mx[d]).sum(), rtol=1e-6,
                                   atol=1e-30)
