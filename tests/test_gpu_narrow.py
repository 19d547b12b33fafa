"""Plans of small images run narrow tiles, the engine the pipelined passes; the
bits are the same.  Shapes: every length of the narrow passes as a row and as
a column length, partial last tiles, the last size that uses them and sizes where
only one of the two passes does.
"""
import numpy as np
import pytest

import imresh_b200 as imr

pytestmark = pytest.mark.gpu

SHAPES = [(64, 64), (65, 64), (64, 68), (3, 128), (128, 4), (192, 100), (100, 192), (1, 256), (256, 260), (384, 768),
          (766, 384), (512, 1024), (1024, 512), (1024, 1024), (1025, 64), (64, 1028), (768, 300)]


@pytest.mark.parametrize("shape", SHAPES)
def test_plan_equals_engine_bit_for_bit(cuda, shape):
    import torch
    H, W = shape
    rng = np.random.default_rng(H * 4099 + W)
    mod = np.abs(rng.standard_normal(shape)).astype(np.float32)
    mod[rng.random(shape) < 0.3] = 0
    p = imr.Params(2, imr.FLT_MIN, 0, 0, 0, 0, 0, 3)
    e = imr.Engine()
    want = e.submit(mod, p)
    e.run()
    assert e.poll()[0]["status"] == 0
    e.close()
    d = torch.from_numpy(mod).cuda()
    got = torch.empty_like(d)
    plan = imr.Plan(W, H, p)
    for _ in range(2):   # the second run starts from the first one's state
        plan.execute(d, got)
        assert np.array_equal(got.cpu().numpy(), want)
    plan.close()
