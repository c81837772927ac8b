"""The quarter-turn orbits of the grid likelihoods (host side, on the CPU):
every pixel once, its orbit's places and radius, the groups' radius spans, and
no tables for pixels that are not whole orbits."""
import numpy as np
import pytest
import torch


def _tables(size, prec, pixels, qrad):
    adj = pytest.importorskip('rspi.adjoint')
    t = lambda a, d=torch.float64: torch.as_tensor(np.ascontiguousarray(a)).to(d)  # noqa: E731
    return adj._orbit_tables(size, prec, pixels, np.arange(pixels.size), qrad, t)


@pytest.mark.parametrize('size', [9, 10, 17, 64, 101])
@pytest.mark.parametrize('prec,tile', [(0, 512), (1, 256)])
def test_orbits(size, prec, tile):
    from rspi import geometry
    _, _, qrad, mask, _ = geometry.phaser_qvals(size)
    px, c = np.flatnonzero(mask), size // 2
    order, xy, rad, rad_q, span = _tables(size, prec, px, qrad[px])
    order, xy, rad, rad_q = (a.numpy() for a in (order, xy, rad, rad_q))
    assert np.array_equal(np.sort(order.ravel()), np.arange(px.size))
    x, y = xy >> 16, xy & 0xffff
    assert x.min() >= 1 and y.min() >= 0
    for k, (u, v) in enumerate(((x, y), (-y, x), (-x, -y), (y, -x))):
        assert np.array_equal(px[order[:, k]], (u + c) * size + v + c)
        np.testing.assert_allclose(qrad[px[order[:, k]]], rad_q[rad], rtol=1e-15)
    spans = [np.ptp(rad[i:i + tile]) + 1 for i in range(0, rad.size, tile)]
    assert span == max(spans)


def test_not_whole_orbits():
    from rspi import geometry
    size = 20
    px = np.flatnonzero(geometry.phaser_qvals(size)[3])
    assert _tables(size, 0, px[1:], np.ones(px.size - 1)) is None
    edge = np.sort(np.append(px, 10))     # a pixel at -c, whose opposite is off the detector
    assert _tables(size, 0, edge, np.ones(edge.size)) is None
    assert _tables(size, 0, px[:0], np.ones(0)) is None
    assert _tables(10 ** 6, 0, px, np.ones(px.size)) is None
