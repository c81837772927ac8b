"""The device-wide exclusive scan (rspi_scan_rows) at the edges of its tiles
(4,096 counts) and of its one-CTA form (four tiles)."""
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize('n', [1, 3, 4095, 4096, 4097, 4 * 4096, 4 * 4096 + 1, 1025 * 4096 + 5])
def test_scan_rows(n):
    from rspi.device import cur_stream, ptr
    from rspi.lib import call
    gen = torch.Generator('cuda').manual_seed(n)
    # totals beyond 32 bits at the largest size
    cnt = torch.randint(0, 1 << 20, (n,), generator=gen, device='cuda', dtype=torch.int32)
    off = torch.full((n + 1,), -1, dtype=torch.int64, device='cuda')
    call('rspi_scan_rows', ptr(cnt), n, ptr(off), cur_stream())
    want = torch.zeros(n + 1, dtype=torch.int64, device='cuda')
    want[1:] = torch.cumsum(cnt.long(), 0)
    assert torch.equal(off, want)
