"""The dispatch rules on sizes (imresh_b200/csrc/rules.hpp), compiled on the CPU, at
the shapes they were measured at; and results on both sides of each line."""
import os
import subprocess

import numpy as np
import pytest

import imresh_b200 as imr

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "imresh_b200", "csrc")


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    def run(expr):
        d = tmp_path_factory.mktemp("rules")
        src, exe = os.path.join(d, "r.cpp"), os.path.join(d, "r")
        with open(src, "w") as f:
            f.write('#include <stdio.h>\n#include "rules.hpp"\nint main() { printf("%%ld", (long)(imr::%s)); }\n' % expr)
        subprocess.run(["g++", "-std=c++17", "-I", CSRC, src, "-o", exe], check=True)
        return int(subprocess.run([exe], check=True, capture_output=True, text=True).stdout)
    return run


def _check_fft(h, w, sign):
    import torch
    rng = np.random.default_rng(h * 4 + w)
    x = (rng.standard_normal((h, w)) + 1j * rng.standard_normal((h, w))).astype(np.complex64)
    d = torch.from_numpy(x.copy()).cuda()
    imr.fft2d(d, w, h, sign)
    xd = x.astype(np.complex128)
    ref = np.fft.fft2(xd) if sign < 0 else np.fft.ifft2(xd) * x.size
    assert np.linalg.norm(d.cpu().numpy() - ref) / np.linalg.norm(ref) < 1e-5   # the transforms' bar


# inverse transforms as measured: column blocks, resident, row blocks, resident, start early
@pytest.mark.parametrize("cols,cres,rows,rres,early", [
    (96, 148, 256, 740, 0),      # 384 x 2048: 15.9 us, early 22.4
    (256, 888, 192, 444, 0),     # 4096 x 192: 15.9, 18.9
    (128, 148, 512, 888, 0),     # 512 x 2048: 13.4, 15.0
    (32, 148, 128, 888, 0),      # 128 x 2048: 10.4, 10.7
    (64, 888, 64, 592, 1),       # 256 x 256: 5.2, 4.9
    (128, 592, 128, 888, 1),     # 512 x 512: 6.25, 5.9
    (512, 444, 768, 444, 1),     # 4096 x 768: 44.2, 43.7
    (192, 148, 700, 592, 1)])
def test_rows_do_not_start_beside_few_column_blocks(rule, cols, cres, rows, rres, early):
    assert rule("fft_rows_start_early(%d, %d, %d, %d)" % (cols, cres, rows, rres)) == early


@pytest.mark.gpu
@pytest.mark.parametrize("h,w", [(2048, 384), (888, 64), (889, 64), (1184, 128), (1185, 128), (192, 4096), (148, 2048), (149, 2048)])
@pytest.mark.parametrize("sign", [-1, 1])
def test_transforms_on_both_sides_of_the_early_start(cuda, h, w, sign):
    _check_fft(h, w, sign)


# grouped rows beside 224 column blocks (896 x 512: 9.2 us, early 8.4); powers of two both ways
@pytest.mark.parametrize("args,early", [("224, 592, 256, 444, true", 1), ("256, 592, 256, 740, true", 1), ("96, 148, 256, 740, false", 0)])
def test_rows_that_do_not_crowd_start_early(rule, args, early):
    assert rule("fft_rows_start_early(%s)" % args) == early


# column blocks of a small plan: 384 x 1024 started early 16.3 us an iteration, in turn 14.5
@pytest.mark.parametrize("blocks,threads,early", [(96, 256, 0), (64, 256, 1), (128, 256, 1), (96, 128, 1), (192, 512, 1)])
def test_half_sm_column_blocks_do_not_pair_up(rule, blocks, threads, early):
    assert rule("small_plan_columns_early(%d, %d)" % (blocks, threads)) == early


# (W, H, wide tile of H, narrow): images with many wide tiles keep them
@pytest.mark.parametrize("w,h,tile,narrow", [(256, 256, 16, 1), (512, 1024, 8, 1), (1168, 512, 16, 1), (1169, 512, 16, 0),
                                             (1024, 1024, 8, 0), (2048, 512, 16, 0), (4096, 128, 16, 0)])
def test_narrow_columns_where_wide_tiles_leave_sms_idle(rule, w, h, tile, narrow):
    assert rule("fft_narrow_columns(%d)" % ((w + tile - 1) // tile)) == narrow


# wide tiles, as many at the same time: 1536 x 1024 26.1 us wide, 24.8 narrow; 1920 x 1024 25.6, 27.2
@pytest.mark.parametrize("tiles,resident,narrow", [(148, 148, 0), (149, 148, 1), (192, 148, 1), (222, 148, 1), (223, 148, 0), (192, 740, 0)])
def test_narrow_columns_where_wide_tiles_begin_a_second_wave(rule, tiles, resident, narrow):
    assert rule("fft_narrow_columns(%d, %d)" % (tiles, resident)) == narrow


@pytest.mark.gpu
@pytest.mark.parametrize("h,w", [(1024, 1185), (1024, 1778), (512, 3072)])
@pytest.mark.parametrize("sign", [-1, 1])
def test_transforms_in_the_second_wave(cuda, h, w, sign):
    _check_fft(h, w, sign)


@pytest.mark.gpu
@pytest.mark.parametrize("h,w", [(64, 33), (128, 3), (128, 1165), (128, 1169), (512, 1168), (512, 1171), (1024, 583), (1024, 585)])
@pytest.mark.parametrize("sign", [-1, 1])
def test_transforms_on_both_sides_of_the_narrow_columns(cuda, h, w, sign):
    _check_fft(h, w, sign)


# an iteration of 2048 x 1024: 38.1 us, rows that start early 39.8
@pytest.mark.parametrize("w,dependent", [(64, 1), (1536, 1), (2048, 0), (4096, 0)])
def test_long_pipelined_rows_do_not_start_early(rule, w, dependent):
    assert rule("pipelined_rows_dependent(%d)" % w) == dependent


# rows of a blur: W, H, taps, 16-byte pieces, rolling kernel (measured us: rolling, other)
@pytest.mark.parametrize("w,h,taps,vec,rolling", [
    (64, 64, 19, 1, 0),          # 4.2, 2.2
    (256, 256, 19, 1, 0),        # 4.5, 2.5
    (16, 1024, 59, 1, 0),        # 5.9, 3.2
    (331, 2649, 5, 0, 0),        # 7.8, 6.8
    (1021, 733, 19, 0, 1),       # 6.0, 8.1
    (64, 16384, 3, 1, 1),        # 7.6, 16.6
    (1000, 800, 19, 1, 1),       # 5.6, 9.0
    (2048, 1536, 19, 1, 1),      # 14, 26
    (4100, 1000, 59, 1, 1)])     # 35, 82
def test_rolling_row_blur_where_its_long_code_pays(rule, w, h, taps, vec, rolling):
    assert rule("hblur_rolling(%d, %d, %d, %d)" % (w, h, taps, vec)) == rolling


@pytest.mark.gpu
@pytest.mark.parametrize("h,w", [(16384, 64), (5003, 61), (4000, 30), (600, 256), (297, 1000), (593, 331), (3479, 463),
                                 (2003, 1023), (7, 4100), (2, 9002), (2, 53952), (2, 53956), (1, 58048)])
@pytest.mark.parametrize("sigma", [0.4, 3.0])
def test_rows_of_a_blur_bitexact(cuda, h, w, sigma):
    """Many narrow rows per block, rows with and without a stage for their sums."""
    import torch

    import oracle
    img = np.random.default_rng(h + w).random((h, w)).astype(np.float32)
    d = torch.from_numpy(img).cuda()
    imr.gaussian_blur(d, None, w, h, sigma, 1)
    assert np.array_equal(d.cpu().numpy(), oracle.blur(img, sigma, "h"))


# an iteration of 128 x 1792: 18.9 us with tiles of two columns, 26.5 with four
@pytest.mark.parametrize("n,w,few", [(1280, 64, 1), (1792, 128, 1), (2000, 222, 1), (2000, 223, 0), (1000, 64, 0), (1920, 1080, 0)])
def test_two_columns_a_tile_for_few_long_columns(rule, n, w, few):
    assert rule("mx_few_columns(%d, %d)" % (n, w)) == few


@pytest.mark.gpu
@pytest.mark.parametrize("h,w", [(1050, 1), (1715, 3), (1792, 128), (2000, 221), (2000, 222), (1458, 223)])
def test_few_long_columns_equal_the_engine_bit_for_bit(cuda, h, w):
    """A plan's tiles of two columns against the engine's tiles of four."""
    rng = np.random.default_rng(h + w)
    mod = np.abs(rng.standard_normal((h, w))).astype(np.float32)
    mod[rng.random((h, w)) < 0.3] = 0
    p = imr.Params(2, imr.FLT_MIN, 0, 0, 0, 0, 0, 3)
    e = imr.Engine()
    want = e.submit(mod, p)
    e.run()
    assert e.poll()[0]["status"] == 0
    e.close()
    plan = imr.Plan(w, h, p)
    assert np.array_equal(plan.execute_host(mod), want)
    plan.close()
    for sign in (-1, 1):
        _check_fft(h, w, sign)


# columns of a blur: tiles of 128 rows, 32 rows instead (us: 32 rows, 128)
@pytest.mark.parametrize("tiles,small", [(32, 1), (160, 1), (174, 1), (188, 0), (256, 0)])   # 188: 8.5, 7.8; 256: 8.1, 6.9
def test_small_blur_tiles_only_where_large_ones_leave_sms_idle(rule, tiles, small):
    assert rule("vblur_small_tiles(%d)" % tiles) == small


@pytest.mark.gpu
@pytest.mark.parametrize("h,w", [(700, 900), (500, 1500), (4095, 199)])
@pytest.mark.parametrize("sigma", [0.4, 10.0])
def test_columns_of_a_blur_bitexact(cuda, h, w, sigma):
    import torch

    import oracle
    img = np.random.default_rng(h + w).random((h, w)).astype(np.float32)
    d = torch.from_numpy(img).cuda()
    imr.gaussian_blur(d, torch.empty_like(d), w, h, sigma, 2)
    assert np.array_equal(d.cpu().numpy(), oracle.blur(img, sigma, "v"))


# numbers, shift: 4096^2 numbers in the smallest chunks took 181 us, 137 at shift 3
@pytest.mark.parametrize("n,shift", [(1, 0), (512 * 384, 0), (2048 * 2048, 0), (8 << 20, 1), (4096 * 4096, 3), (32 << 20, 1)])
def test_chunks_of_a_large_random_field(rule, n, shift):
    assert rule("rand_chunk_shift(%d)" % n) == shift


@pytest.mark.gpu
@pytest.mark.parametrize("n", [6999999, 7000001, 14000001, 148 * 128 * 992, 148 * 128 * 992 + 1])
def test_random_field_bitexact_on_both_sides_of_its_chunks(cuda, n):
    import torch

    import oracle
    d = torch.empty(n, dtype=torch.complex64, device="cuda")
    imr.rand_field(d, n, 7)
    got = d.cpu().numpy()
    np.testing.assert_array_equal(got.real, oracle.rand_field(n, 7))
    assert not got.imag.any()
