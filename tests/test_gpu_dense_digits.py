"""Digit planes of the dense form's log-slices: the paired and the plain
slices give the same bytes, which are those of the FP64 rotated slice's
fixed-point value, for row ranges inside a state's rotations."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('size,n_sel,states,num_rot,r0,r1', [
    (21, 1, 1, 1, 0, 1), (21, 127, 3, 4, 1, 11), (37, 300, 9, 3, 0, 27), (38, 384, 17, 5, 7, 84)])
def test_digits_of_pairs_and_plain_slices(size, n_sel, states, num_rot, r0, r1):
    from rspi.device import cur_stream, ptr
    from rspi.lib import call
    rng = np.random.default_rng(size + n_sel)
    npix = size * size
    dev = torch.device('cuda')
    holo = torch.from_numpy(np.exp(rng.normal(0., 3., (states, npix)))).to(dev)
    holo[:, ::7] = 0.                                 # the sentinel
    pairs = torch.empty((states, npix, 2), dtype=torch.float64, device=dev)
    call('rspi_holo_pairs', ptr(holo), states, size, ptr(pairs), cur_stream())
    ang = np.arange(num_rot) * np.pi / num_rot
    rot = torch.from_numpy(np.stack([np.cos(ang), np.sin(ang)], 1).ravel()).to(dev)
    bg = torch.zeros(npix, dtype=torch.float64, device=dev)
    sel = torch.from_numpy(np.sort(rng.choice(npix, n_sel, replace=False)).astype(np.int32)).to(dev)
    k_pad = -(-n_sel // 128) * 128
    rows = r1 - r0
    out = []
    for name, src in (('rspi_rot_log_fixed', holo), ('rspi_rot_log_fixed_pairs', pairs)):
        d = torch.full((4, rows + 1, k_pad), 77, dtype=torch.uint8, device=dev)
        err = torch.zeros(1, dtype=torch.int32, device=dev)
        call(name, ptr(src), states, num_rot, ptr(rot), size, ptr(bg), ptr(sel), n_sel, k_pad,
             r0, r1, rows + 1, ptr(d), ptr(err), cur_stream())
        assert int(err.item()) == 0
        out.append(d.cpu().numpy())
    assert np.array_equal(out[0], out[1])
    assert np.all(out[0][:, rows] == 77)              # no row beyond the range
    p_row = -(-n_sel // 32) * 32 + 32
    lsl = torch.empty((rows, p_row), dtype=torch.float64, device=dev)
    amax = torch.zeros(1, dtype=torch.float32, device=dev)
    call('rspi_rot_log_slices_pairs', ptr(pairs), states, num_rot, ptr(rot), size, ptr(bg),
         ptr(sel), n_sel, p_row, r0, r1, ptr(lsl), 1, ptr(amax), cur_stream())
    want = np.rint(lsl.cpu().numpy()[:, :n_sel] * 2. ** 21).astype(np.int64)
    d = out[0][:, :rows].astype(np.int64)
    got = d[0] + (d[1] << 8) + (d[2] << 16) + (d[3].astype(np.uint8).view(np.int8).astype(np.int64) << 24)
    assert np.array_equal(got[:, :n_sel], want)
    assert not got[:, n_sel:].any()
