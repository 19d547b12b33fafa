"""Bluestein transforms at the edges of their work lengths (256 .. 4096): the
smallest and the largest length of each, as rows and as columns, with partial
last tiles.  Tolerance: the per-kernel bar of the transforms, 1e-5 relative
L2 against numpy's FP64 transform.
"""
import numpy as np
import pytest

import imresh_b200 as imr

pytestmark = pytest.mark.gpu

LENGTHS = [67, 127, 131, 255, 257, 511, 514, 1023, 1027, 2047]


@pytest.mark.parametrize("n", LENGTHS)
@pytest.mark.parametrize("other", [3, 17])
@pytest.mark.parametrize("rows", [True, False])
@pytest.mark.parametrize("sign", [-1, 1])
def test_bluestein_lengths_match_fp64(cuda, n, other, rows, sign):
    import torch
    shape = (other, n) if rows else (n, other)
    rng = np.random.default_rng(n * 4 + other)
    x = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)
    d = torch.from_numpy(x.copy()).cuda()
    imr.fft2d(d, shape[1], shape[0], sign)
    y = d.cpu().numpy()
    xd = x.astype(np.complex128)
    ref = np.fft.fft2(xd) if sign < 0 else np.fft.ifft2(xd) * x.size
    assert np.linalg.norm(y - ref) / np.linalg.norm(ref) < 1e-5
