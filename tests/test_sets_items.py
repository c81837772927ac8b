"""Entries of several photons and the pieces of long sets of the frame-set
kernel: the layouts hold every photon once, and the likelihoods lie within
the screening bound of the FP64 form's, with its rescored results."""
import numpy as np
import pytest
import torch

from rspi import device


@pytest.mark.parametrize('parts,n_sets', [(1, 1), (1, 7), (2, 126), (4, 3), (3, 700), (2, 64)])
def test_items_cover_the_sets(parts, n_sets):
    """Every set's groups, and each quarter warp's, once and in order; only
    the first SPLIT_SETS sets are cut; the pieces of a part have slots of
    their own; a set's items are in its queue."""
    gen = torch.Generator().manual_seed(parts * 1000 + n_sets)
    g = (torch.rand(parts, n_sets, generator=gen) ** 6 * 400).to(torch.int32)
    g = torch.sort(g, 1, descending=True).values.reshape(-1)
    g[0] += 50 * n_sets                        # one long set
    g[-1] = 0 if n_sets > 1 else g[-1]         # an empty one
    q = (g[:, None] - torch.randint(0, 4, (g.numel(), 4), generator=gen)).clamp(min=0)
    q[:, 1] = g
    goff = torch.cat([torch.zeros(1, dtype=torch.int64), g.long().cumsum(0)])
    items, off, slots = device.EStep._sets_items(g, q.to(torch.int32).reshape(-1), goff, parts,
                                                 n_sets)
    queues = 4 if parts > 1 else 1
    assert slots > 1 and off[0] == 0 and int(off[-1]) == items.shape[0]
    got = {}
    for h in range(parts):
        used = []
        for k in range(queues):
            for i in range(int(off[h * queues + k]), int(off[h * queues + k + 1])):
                s, g0, n, info, *quarter = items[i].tolist()
                base, piece, pieces = info & 0xffff, info >> 16 & 255, info >> 24
                assert s % queues == k and piece < pieces <= 127
                if pieces > 1:
                    assert s < device.SPLIT_SETS and n > 0 and base + piece < slots
                    used.append(base + piece)
                got.setdefault((h, s), []).append((piece, g0, n, quarter, pieces))
        assert len(used) == len(set(used))
    assert len(got) == parts * n_sets
    for (h, s), it in got.items():
        it.sort()
        j = h * n_sets + s
        assert [x[0] for x in it] == list(range(it[0][4]))
        assert it[0][1] == int(goff[j])
        assert all(a[1] + a[2] == b[1] for a, b in zip(it, it[1:]))
        assert it[-1][1] + it[-1][2] == int(goff[j + 1])
        # a quarter warp's groups: whole pieces, then a remainder, then none
        left = q[j].tolist()
        for _, _, n, quarter, _ in it:
            assert quarter == [min(n, x) for x in left]
            left = [x - y for x, y in zip(left, quarter)]
        assert left == [0] * 4


def test_few_groups_are_not_cut():
    g = torch.full((2 * 40,), 9, dtype=torch.int32)
    goff = torch.arange(81) * 9
    assert device.EStep._sets_items(g, g.repeat_interleave(4), goff, 2, 40) == (None, None, 0)


def _data(n, mean):
    from test_gpu_estep import E, random_photons
    size = 37
    d = random_photons(size, n, mean * size, 15, empty_frames=(2, 9), heavy=5)
    ds = E.parse_photons(d['ones'], d['multi'], d['place_ones'], d['place_multi'],
                         d['count_multi'], size * size, False)
    states = E.generate_states(E.parse_triple('0 0 1'), E.parse_triple('0 0 1'),
                               E.parse_triple('2 3 2'))
    return size, ds, states


@pytest.mark.gpu
@pytest.mark.parametrize('n,parts', [(61, 1), (300, 2), (45, 3), (33, 4)])
def test_counted_entries_hold_the_photons(n, parts):
    """A pixel of k photons as floor(k / 8) entries of 8 and the binary
    digits of the rest, in its frame's lane and part; a quarter warp's eight
    lanes read eight bank classes at every step."""
    from test_gpu_estep import _estep, _photons, frame_photons16
    size, ds, (sx, sy, dia, _) = _data(n, 40.)
    es = _estep(_photons(ds, False), size, 3, sx, sy, dia, ds['bg'], form='screen',
                screen_parts=parts)
    w = es.wide
    assert w['counted'] and w['n_parts'] == parts
    pw, ns = w['part_w'], w['n_sets']
    ent = w['entries'].cpu().numpy().view(np.uint16).reshape(-1, 32, 4).astype(np.int64)
    goff, sf = w['group_off'].cpu().numpy(), w['set_frames'].cpu().numpy()
    qg = w['quarter_groups'].cpu().numpy()
    photons = frame_photons16(es)
    for s in range(ns):
        for h in range(parts):
            blk = ent[goff[h * ns + s]:goff[h * ns + s + 1]].transpose(0, 2, 1).reshape(-1, 32)
            col, cnt = blk & 0x3fff, 1 << (blk >> 14)
            assert np.all(col <= pw + 7)
            for q in range(4):
                steps = 4 * qg[(h * ns + s) * 4 + q]
                cls = np.sort(col[:steps, 8 * q:8 * q + 8] % 8, 1)
                assert np.all(cls == np.arange(8))
                assert np.all(col[steps:, 8 * q:8 * q + 8] >= pw)
            for lane in range(32):
                fr = sf[32 * s + lane]
                real = col[:, lane] < pw
                if fr < 0:
                    assert not real.any()
                    continue
                k = np.bincount(photons[fr][photons[fr] // pw == h] % pw, minlength=pw)
                got = np.bincount(col[real, lane], weights=cnt[real, lane], minlength=pw)
                assert np.array_equal(got, k)
                assert real.sum() == sum(int(x) // 8 + bin(int(x) % 8).count('1') for x in k)


@pytest.mark.gpu
@pytest.mark.parametrize('named', [False, True])
@pytest.mark.parametrize('shares', [0, 3, 10 ** 9])
@pytest.mark.parametrize('n,parts,warps', [(1, 1, 1), (61, 1, 32), (300, 2, 16), (45, 3, 7),
                                           (2300, 2, 32)])
def test_counted_and_cut_sets_within_the_bound(n, parts, warps, shares, named, monkeypatch):
    """Counted or single entries (kernel asked for by name), sets whole, cut
    by the rule or all cut: the candidate threshold's bound eps_d = 2^-24
    ((rows_d + 8) photons_d lmax + |L|) against the FP64 form, and its
    rescored argmax, maximum and log-sum-exp."""
    from test_gpu_estep import _estep, _photons
    monkeypatch.setattr(device, 'SPLIT_SHARES', shares)
    size, ds, (sx, sy, dia, _) = _data(max(n, 10), 40.) if n > 1 else _data(10, 4.)
    rng = np.random.default_rng(n)
    model = torch.from_numpy(rng.random(size * size) + 1j * rng.random(size * size)).cuda()
    ref = _estep(_photons(ds, False), size, 5, sx, sy, dia, ds['bg'], form='fp64')
    ref.run(model)
    want_r = [t.cpu().numpy() for t in ref.reduce()]
    want = ref.frame_prob().cpu().numpy()
    ph = _photons(ds, False)
    kw = dict(kernel='sets') if named else {}
    es = _estep(ph, size, 5, sx, sy, dia, ds['bg'], form='screen', states_per_tile=4,
                warps=warps, screen_parts=parts, **kw)
    if named:
        assert not es.wide['counted']
    assert (es.wide['seg_slots'] > 0) == (shares == 0) or shares == 3
    for _ in range(2):                       # twice: the pieces' counters start anew
        es.run(model)
        got_r = [t.cpu().numpy() for t in es.reduce()]
    ph.err.check('frame-set kernel')
    got = es.frame_prob().cpu().numpy().astype(np.float64)
    rows = np.diff(es._eps_rows().cpu().numpy()).astype(np.float64)
    phot = es.ll['frame_sel_photons'].cpu().numpy().astype(np.float64)
    lmax = float(es.lmax.cpu().numpy().reshape(-1)[0])
    eps = 2. ** -24 * ((rows + 8.) * phot * lmax + np.abs(want) + 1.)
    fin = np.isfinite(want)
    assert np.array_equal(fin, np.isfinite(got))
    assert np.all(np.abs(np.where(fin, got - want, 0.)) <= np.where(fin, eps, 0.))
    assert np.array_equal(got_r[1], want_r[1])
    np.testing.assert_allclose(got_r[0], want_r[0], rtol=1e-14)
    np.testing.assert_allclose(got_r[2], want_r[2], rtol=1e-12)
