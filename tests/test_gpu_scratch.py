"""The memory that synchronous host calls keep is not lost to others."""
import numpy as np
import pytest

import imresh_b200 as imr

pytestmark = pytest.mark.gpu


def _budget():
    e = imr.Engine()
    b = e.info()["device_bytes_budget"]
    e.close()
    return b


def test_engine_counts_kept_scratch_as_free(cuda):
    import torch
    torch.cuda.synchronize()
    obj = np.random.default_rng(0).random((2048, 2048)).astype(np.float32)   # 50 MB of scratch
    imr.diffraction_intensity(obj)   # (tables and context memory are there)
    imr.release_scratch()
    before = _budget()
    imr.diffraction_intensity(obj)
    assert abs(_budget() - before) < 8 << 20


def test_release_gives_the_scratch_back(cuda):
    import torch
    obj = np.random.default_rng(1).random((2048, 2048)).astype(np.float32)
    want = imr.diffraction_intensity(obj)
    imr.release_scratch()
    free = torch.cuda.mem_get_info()[0]
    assert np.array_equal(imr.diffraction_intensity(obj), want)   # and it is taken again
    assert torch.cuda.mem_get_info()[0] <= free - (32 << 20)
    imr.release_scratch()
    assert torch.cuda.mem_get_info()[0] >= free - (2 << 20)
