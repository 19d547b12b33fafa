"""Lengths without a compile-time kernel: the grouped-pass transforms.

Shapes cover every pass of one or two radices, one row and one column, tiles
with a partial last tile, both widths of the column block (up to 1024 rows and
above) and the longest rows.  Tolerance: the per-kernel bar of the transforms,
1e-5 relative L2 against numpy's FP64 transform.
"""
import numpy as np
import pytest

import imresh_b200 as imr

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (1, 7), (3, 1), (2, 2), (32, 16), (10, 12), (14, 18), (21, 15), (45, 35), (9, 441), (5, 1701),
          (1024, 45), (1029, 6), (1120, 9), (1792, 5), (2000, 3), (3, 2000), (300, 600)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("sign", [-1, 1])
def test_grouped_fft_matches_fp64(cuda, shape, sign):
    import torch
    rng = np.random.default_rng(shape[0] * 4099 + shape[1])
    x = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)
    d = torch.from_numpy(x.copy()).cuda()
    imr.fft2d(d, shape[1], shape[0], sign)
    y = d.cpu().numpy()
    xd = x.astype(np.complex128)
    ref = np.fft.fft2(xd) if sign < 0 else np.fft.ifft2(xd) * x.size
    assert np.linalg.norm(y - ref) / np.linalg.norm(ref) < 1e-5


def test_grouped_sizes_share_engine_launches(cuda):
    """Jobs of different lengths in one launch of the same kernel: each tile
    needs its own job's shared memory, table and schedule; bit-identical to
    the plan alone."""
    import torch
    rng = np.random.default_rng(3)
    shapes = [(1000, 60), (20, 300), (300, 20), (1120, 12), (60, 1000), (63, 105)]
    p = imr.Params(2, imr.FLT_MIN, 0, 0, 0, 0, 0, 3)
    mods = [np.abs(rng.standard_normal(s)).astype(np.float32) for s in shapes]
    e = imr.Engine()
    outs = [e.submit(m, p, tag=i) for i, m in enumerate(mods)]
    e.run()
    assert all(r["status"] == 0 for r in e.poll())
    e.close()
    for m, o in zip(mods, outs):
        d = torch.from_numpy(m).cuda()
        r = torch.empty_like(d)
        plan = imr.Plan(m.shape[1], m.shape[0], p)
        plan.execute(d, r)
        torch.cuda.synchronize()
        assert np.array_equal(o, r.cpu().numpy())
        plan.close()
