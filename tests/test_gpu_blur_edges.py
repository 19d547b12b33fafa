"""The blur where its tiles end: rows longer than one round of a block, several
short rows per block, widths and buffers that 16-byte loads do not fit, few and
many taps.  Bit-exact against the oracle's blur (same tap order, separate
multiply and add).
"""
import numpy as np
import pytest

import imresh_b200 as imr
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1), (2, 17), (5, 4096), (3, 4097), (2, 9000), (900, 12), (129, 33), (131, 64)])
@pytest.mark.parametrize("sigma", [0.3, 3.0, 10.0])
@pytest.mark.parametrize("offset", [0, 1])
def test_blur_bitexact_at_tile_edges(cuda, shape, sigma, offset):
    import torch
    H, W = shape
    img = np.random.default_rng(H * 4099 + W).random(shape).astype(np.float32)
    for axes, axis in ((1, "h"), (2, "v"), (3, "hv")):
        buf = torch.empty(2, H * W + offset, device="cuda")
        d, tmp = buf[0, offset:], buf[1, offset:]   # the second buffer's alignment follows from the first's length
        d.copy_(torch.from_numpy(img).cuda().reshape(-1))
        imr.gaussian_blur(d, tmp, W, H, sigma, axes)
        assert np.array_equal(d.cpu().numpy().reshape(shape), oracle.blur(img, sigma, axis)), axis
