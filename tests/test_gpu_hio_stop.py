"""Fixed-support HIO that stops in the middle of a run, and mask bytes other than
0 and 1, for each kind of pass: narrow, pipelined, grouped and chirp-z rows; column
passes that form the error beside their tiles (narrow, grouped, chirp-z) and ones
that leave it to the rows.  Checked against the oracle.

Tolerances: the error of an iteration within 1e-4, or 10 times the oracle's own
float-against-64-bit distance where HIO already amplifies rounding; the output as
tests/test_gpu_hio.py; the iteration exactly.
"""
import numpy as np
import pytest

import imresh_b200 as imr
import oracle

from .test_gpu_hio import _assert_close_to_oracle, _case

pytestmark = pytest.mark.gpu

# (H, W): grouped both ways; chirp-z both ways; narrow rows and columns that do not
# defer (chirp-z below 256); 500 column tiles; chirp-z columns of pipelined rows;
# grouped columns of pipelined rows; narrow; chirp-z rows and pipelined columns
SHAPES = [(60, 300), (300, 60), (97, 101), (61, 64), (100, 2000), (1028, 128), (1280, 64), (64, 192), (128, 1028)]


def _check_errors(errs, ref, ref64):
    tol = np.maximum(1e-4, 10 * np.abs(ref / ref64 - 1))
    assert (np.abs(errs / ref - 1) <= tol).all(), (errs, ref)


@pytest.mark.parametrize("shape", SHAPES)
def test_stop_in_the_middle_of_a_run(cuda, shape):
    H, W = shape
    M, mask = _case(H, W, seed=5)
    errs = oracle.hio(M, mask, 24, 1e-30, 0.9).errors
    k = next(k for k in range(5, 24) if errs[k] < 0.98 * errs[:k].min())
    target = float(0.5 * (errs[k] + errs[:k].min()))
    ref = oracle.hio(M, mask, 24, target, 0.9)
    ref64 = oracle.hio(M, mask, k, 1e-30, 0.9, fp64=True)
    assert ref.iterations == k
    plan = imr.HioPlan(W, H, 24, target, 0.9)
    for _ in range(2):   # the second run starts from the stopped one's state
        out = plan.execute_host(M, mask)
        iters, last, got = plan.stats()
        assert iters == k
        assert last < target and last == got[k]
        _check_errors(got[:k + 1], ref.errors[:k + 1], ref64.errors[:k + 1])
        _assert_close_to_oracle(out, ref.out, M, mask, k)
    plan.close()


@pytest.mark.parametrize("shape", [(64, 64), (2048, 64), *SHAPES])
def test_mask_bytes_weigh_the_error(cuda, shape):
    """Bytes 0, 1, 2 and 255: a byte of 1 keeps a pixel in the feedback, the error is
    weighted with the byte."""
    H, W = shape
    M, mask = _case(H, W, seed=5)
    mask = mask.copy()
    pick = np.random.default_rng(H + W).random(mask.shape)
    mask[pick < 0.2] = 2
    mask[pick > 0.9] = 255
    assert set(np.unique(mask)) == {0, 1, 2, 255}
    n = 3
    ref = oracle.hio(M, mask, n, 1e-30, 0.9)
    ref64 = oracle.hio(M, mask, n, 1e-30, 0.9, fp64=True)
    plan = imr.HioPlan(W, H, n, 1e-30, 0.9)
    out = plan.execute_host(M, mask)
    iters, _, got = plan.stats()
    plan.close()
    assert iters == ref.iterations == n
    _check_errors(got[:n + 1], ref.errors[:n + 1], ref64.errors[:n + 1])
    _assert_close_to_oracle(out, ref.out, M, mask, n)
