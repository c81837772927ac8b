"""Digit planes of the dense form's log-slices where CTAs share the columns:
the values of test_gpu_dense_digits around a part's 1,024 columns, and eight
states of one rotation in about the time of one."""
import numpy as np
import pytest
import torch

import test_gpu_dense_digits as digits

pytestmark = pytest.mark.gpu


# columns: one part, a column more, one short of two, several; rows: one, and
# ranges that cut a state's rotations
@pytest.mark.parametrize('n_sel,states,num_rot,r0,r1', [
    (1024, 1, 1, 0, 1), (1025, 9, 2, 1, 17), (2047, 3, 4, 2, 11), (3700, 8, 1, 0, 8),
    (3600, 17, 3, 7, 50)])
def test_digits_in_column_parts(n_sel, states, num_rot, r0, r1):
    digits.test_digits_of_pairs_and_plain_slices(61, n_sel, states, num_rot, r0, r1)


def test_few_rows_fill_the_gpu():
    """36,000 columns of one rotation: eight states, one CTA's rows when the
    columns are not shared (over four times one state's time), against one."""
    from rspi.device import cur_stream, ptr
    from rspi.lib import call
    size, states = 215, 8
    npix, dev = size * size, torch.device('cuda')
    pairs = torch.rand((states, npix, 2), dtype=torch.float64, device=dev)
    rot = torch.tensor([np.cos(0.3), np.sin(0.3)], dtype=torch.float64, device=dev)
    bg = torch.zeros(npix, dtype=torch.float64, device=dev)
    n_sel = 36096
    sel = torch.arange(4000, 4000 + n_sel, dtype=torch.int32, device=dev)
    out = torch.empty((4, states, n_sel), dtype=torch.uint8, device=dev)
    err = torch.zeros(1, dtype=torch.int32, device=dev)

    def median_us(rows):
        times = []
        for k in range(14):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            torch.cuda.synchronize()
            a.record()
            call('rspi_rot_log_fixed_pairs', ptr(pairs), states, 1, ptr(rot), size, ptr(bg),
                 ptr(sel), n_sel, n_sel, 0, rows, states, ptr(out), ptr(err), cur_stream())
            b.record()
            torch.cuda.synchronize()
            times.append(1e3 * a.elapsed_time(b))
        return sorted(times[3:])[5]

    assert median_us(8) < 2.5 * median_us(1)
    assert int(err.item()) == 0
