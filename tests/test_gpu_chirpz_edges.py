"""Chirp-z lengths where the work length changes: the smallest length without a
direct transform of each (65, 129, 257, 513, 1025, with the longest padding) beside the
largest of the one before.  Transforms: the per-kernel bar, 1e-5 relative L2 against
numpy's FP64 transform.  Reconstructions: one cycle against the oracle, as
tests/test_gpu_shrinkwrap.py.
"""
import numpy as np
import pytest

import imresh_b200 as imr
import oracle
from imresh_b200 import data

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [65, 127, 129, 255, 257, 511, 513, 1023, 1025, 2047])
@pytest.mark.parametrize("other", [3, 17])
@pytest.mark.parametrize("rows", [True, False])
@pytest.mark.parametrize("sign", [-1, 1])
def test_transforms_match_fp64(cuda, n, other, rows, sign):
    import torch
    shape = (other, n) if rows else (n, other)
    rng = np.random.default_rng(n * 4 + other)
    x = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)
    d = torch.from_numpy(x.copy()).cuda()
    imr.fft2d(d, shape[1], shape[0], sign)
    xd = x.astype(np.complex128)
    ref = np.fft.fft2(xd) if sign < 0 else np.fft.ifft2(xd) * x.size
    assert np.linalg.norm(d.cpu().numpy() - ref) / np.linalg.norm(ref) < 1e-5


@pytest.mark.parametrize("shape", [(65, 129), (129, 65), (257, 127), (127, 257), (513, 64), (64, 513), (1025, 65), (65, 1025)])
def test_one_cycle_matches_oracle(cuda, shape):
    H, W = shape
    M, _ = data.make_modulus(data.BlobSpec(W, H, 12, 0.15 * min(W, H), (1.5, 2.5), (0.5, 1.0), None), 1)
    ref = oracle.shrinkwrap(M, oracle.SwParams(1, imr.FLT_MIN, 0.9, 0.04, 0.2, 3.0, 0.01, 1))
    plan = imr.Plan(W, H, imr.Params(1, imr.FLT_MIN, 0.9, 0.04, 0.2, 3.0, 0.01, 1))
    out = plan.execute_host(M)
    n, errs = plan.stats()
    mask = plan.state("mask")
    plan.close()
    assert n == 1
    assert np.mean(mask != ref.mask) <= 1e-3
    assert np.linalg.norm(out - ref.out) / np.linalg.norm(ref.out) < 1e-4
    assert errs[0] == pytest.approx(ref.errors[0], rel=1e-4)
