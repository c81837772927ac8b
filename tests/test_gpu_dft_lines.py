"""The centred transform at the edges of its line kernel (the shortest lines,
an odd last line, several rounds of outputs, the longest) against NumPy's.
Each output sums n products per axis in FP64: within n 2^-53 of its line's
magnitude sum, far below 1e-12 of the largest output here."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('size', [2, 3, 4, 7, 255, 256, 383, 1024])
@pytest.mark.parametrize('inverse', [0, 1])
def test_centred_transform_edges(size, inverse):
    from rspi.device import cur_stream, ptr
    from rspi.lib import call
    rng = np.random.default_rng(size)
    x = rng.standard_normal((size, size)) + 1j * rng.standard_normal((size, size))
    d = torch.from_numpy(x).cuda()
    out, work = torch.empty_like(d), torch.empty_like(d)
    call('rspi_cdft2', ptr(d), ptr(out), ptr(work), size, inverse, cur_stream())
    fn = np.fft.ifftn if inverse else np.fft.fftn
    want = np.fft.fftshift(fn(np.fft.ifftshift(x)))
    assert np.abs(out.cpu().numpy() - want).max() <= 1e-12 * np.abs(want).max()
