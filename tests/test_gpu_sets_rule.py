"""The layouts that the shipped rules choose: a set far longer than a warp's
share is cut, one that is not stays whole; entries of several photons where
they leave out one entry in COUNT_GAIN or more, single ones elsewhere."""
import numpy as np
import pytest

from oracle import emc_oracle as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('heavy,mean,cut,counted', [
    (40000, 0.02, True, True),       # one frame of many photons per pixel among light ones
    (0, 0.02, False, False),         # 1,300 alike frames, pixels seldom repeat
    (0, 1.5, False, True)])          # 1,300 alike, most pixels repeat
def test_shipped_rules(heavy, mean, cut, counted):
    from rspi.photonfile import sparse_from_dense
    from test_gpu_estep import _estep, _photons
    size, n = 31, 1300               # 41 sets for 32 warps
    rng = np.random.default_rng(4)
    frames = rng.poisson(mean, (n, size * size))
    if heavy:
        frames[7] = rng.poisson(heavy / size ** 2, size * size)
    d = sparse_from_dense(frames)
    ds = E.parse_photons(d['ones'], d['multi'], d['place_ones'], d['place_multi'],
                         d['count_multi'], size * size, True)
    sx, sy, dia, _ = E.generate_states((0., 1., 2), (0., 0., 1), (6., 8., 2))
    es = _estep(_photons(ds, False), size, 3, sx, sy, dia, ds['bg'], form='screen',
                states_per_tile=4)
    assert es.kernel == 'sets'
    assert (es.wide['seg_slots'] > 0) == cut
    assert es.wide['counted'] == counted


@pytest.mark.parametrize('extra', ['', 'kernel = sets\n'])
def test_a_configuration_that_names_the_kernel_keeps_its_layout(extra, tmp_path):
    """`kernel = sets` asks for what is the default anyway: the same entries."""
    from emc import EMC
    from helpers import write_case
    from rspi.photonfile import sparse_from_dense
    size = 31
    rng = np.random.default_rng(5)
    data = dict(sparse_from_dense(rng.poisson(1.5, (40, size * size))),
                num_pix=np.array([size * size]))
    rec = EMC(write_case(str(tmp_path), data=data, size=size, num_rot=3, shiftx='0 1 2',
                         shifty='0 0 1', sphere_dia='6 8 2', need_scaling=True, extra=extra))
    assert rec.estep.kernel == 'sets' and rec.estep.wide['counted']


@pytest.mark.parametrize('mean,pays', [(0.02, False), (1.5, True)])
def test_whether_counts_pay_is_asked_once(mean, pays, monkeypatch):
    """Another tiling (the tuner tries several) rebuilds the entries without
    counting them in both layouts again where the first count rejected one."""
    from rspi import device
    from rspi.photonfile import sparse_from_dense
    from test_gpu_estep import _estep, _photons
    size, n = 31, 70
    d = sparse_from_dense(np.random.default_rng(6).poisson(mean, (n, size * size)))
    ds = E.parse_photons(d['ones'], d['multi'], d['place_ones'], d['place_multi'],
                         d['count_multi'], size * size, True)
    sx, sy, dia, _ = E.generate_states((0., 1., 2), (0., 0., 1), (6., 8., 2))
    es = _estep(_photons(ds, False), size, 3, sx, sy, dia, ds['bg'], form='screen',
                states_per_tile=4)
    assert es.wide['counted'] == pays
    seen = []
    call = device.call
    monkeypatch.setattr(device, 'call', lambda name, *a: (seen.append(name), call(name, *a))[1])
    es.configure(screen_parts=2)
    assert es.wide['counted'] == pays and es.wide['n_parts'] == 2
    assert ('rspi_sets_counts32' in seen) == pays
    assert ('rspi_sets_counts' in seen) == (not pays)
