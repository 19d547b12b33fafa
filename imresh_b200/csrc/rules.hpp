// Rules of the dispatch that depend on sizes only (host code, no CUDA).
#pragma once

namespace imr {

constexpr int kSms = 148;

// Whether the second transform of a plain 2D transform starts while the first one
// drains (programmatic dependent launch).  It takes 0.3-0.6 us off a transform (512 x 512
// 6.25 -> 5.9 us), but blocks that start early go to the SMs that are idle then, several
// each, and stay there.  In an inverse transform the columns come first: a column block
// takes up to a whole SM, and rows that start beside few of them crowd on the others
// (inverse 384 x 2048, 96 column blocks: 15.9 -> 22.4 us; 4096 x 192 15.9 -> 18.9; 512 x 2048
// 13.4 -> 15.0).  So rows start early when they are too few to crowd, when two column
// blocks per SM leave no SM idle, or when they are more than one wave takes.  Row
// blocks are short and small: columns after them gain at every size measured.
// `cols_resident`, `rows_resident`: blocks that run at the same time.  `mixes`: the two
// kinds of blocks were never seen to crowd -- grouped and chirp-z rows (896 x 512 9.2 ->
// 8.4 us, 1920 x 256 9.0 -> 8.4), or powers of two both ways with more than one column
// block to an SM (1024 x 512 8.6 -> 8.2).
inline bool fft_rows_start_early(int cols, int cols_resident, int rows, int rows_resident, bool mixes = false)
{
    return mixes || rows <= 111 || cols >= 2 * kSms || rows > rows_resident || (rows <= kSms && cols_resident > kSms);
}

// Whether the columns of a plain transform run in narrow tiles (4 columns) instead
// of the wide ones (`wide_tiles` of them; 16 columns up to H = 512, 8 at 1024):
// where the wide tiles leave half of the SMs without one.  Whole transform, wide ->
// narrow: 256 x 256 6.2 -> 5.2 us (16 wide tiles), 512 x 1024 10.5 -> 8.9 (64); beyond
// that narrow tiles only make the strides shorter: 2048 x 512 13.0 -> 13.9 (128),
// 2048 x 1024 23.8 -> 25.0 (256), 4096 x 64 7.7 -> 8.0 -- unless the wide ones
// (`wide_resident` of them run at the same time) just begin a second wave:
// 1536 x 1024 (192 on 148) 26.1 -> 24.8, 3072 x 512 26.2 -> 25.0, 1920 x 1024 (240) 25.6 -> 27.2.
inline bool fft_narrow_columns(int wide_tiles, int wide_resident = 1 << 30)
{
    return 2 * wide_tiles < kSms || (wide_tiles > wide_resident && 2 * wide_tiles <= 3 * wide_resident);
}

// Whether the passes of an iteration are launched dependently (launch_pass):
// `tiles` work items on at most `resident` CTAs for each of the two passes.
// It takes 1.1-1.6 us off an iteration (256^2 9.4 -> 8.0 us, 192^2 11.4 -> 10.3,
// 1021 x 733 54.2 -> 51.5), but CTAs that start early go to the SMs that are idle
// then: a pass of one wave that needs all SMs evenly gets several CTAs on some of
// them (1024^2 20.3 -> 22.4, 1000 x 800 35.1 -> 40.5).  So a pass either leaves a
// quarter of the SMs without work, or has more tiles than one wave takes; with
// more than three waves the gap is too small a part to gain (2048^2: 2 % slower).
inline bool dependent_pass(int tiles, int resident)
{
    return tiles <= 111 || (tiles > resident && tiles <= 3 * resident);
}
// Pipelined rows of 2048 and more do not prepare before their wait nor release the
// columns half-way, so an early start gives them nothing, and rows that sit beside
// the columns' last tiles cost 2048 x 1024 38.1 -> 39.8 us (3072 x 512 39.5 and 39.9 the
// other way).
inline bool pipelined_rows_dependent(int W) { return W < 2048; }
// Whether the columns of a small plan start while its narrow rows drain.  A column
// block of 256 threads takes half an SM: more than 64 of them but less than one per SM
// go two to those SMs that are free first, and the others wait for them: 384 x 1024
// (96 blocks) 16.3 us an iteration, in turn 14.5; 384 x 640 between 15.0 and 17.1 from
// run to run, 14.7; 384 x 768 14.3 and 14.6.
inline bool small_plan_columns_early(int blocks, int threads) { return threads < 256 || blocks <= 64 || blocks >= 128; }

// Whether the rows of a Gaussian blur of K taps run the kernel that makes 16
// neighbouring outputs per thread from rolling registers, instead of the one that
// makes one output per thread and turn (256 a turn, one row per CTA).  The rolling
// kernel loads each tap once and takes several rows per CTA, but its code is long and
// runs cold: 64 x 64 takes 3.1 us instead of 2.0, 256 x 256 (19 taps) 4.1 instead of
// 2.5; 1000 x 800 5.6 instead of 9.0, 2048 x 1536 14 instead of 26, 64 x 16384 9.8
// instead of 18.3.  Left side: what it saves, right side: what it costs, in us, a
// least-squares fit of both kernels' times at 200 sizes with 3 to 59 taps (`vec`: rows
// of 16-byte pieces).  On the mean its choice is within 1 % of the faster kernel.
inline bool hblur_rolling(int W, int H, int K, bool vec)
{
    const double turns = (W + 255) / 256, mpx = 1e-6 * W * H;
    return 0.14 * turns + 0.007 * turns * K + 0.54e-3 * H + (0.126 * K - 0.5) * mpx >
           1.05 + 0.02 * K + (vec ? 0.0 : 1.0 + 0.4 * mpx);
}

// Whether grouped-pass columns of n > 1024 values run in tiles of two columns instead
// of four, for an image of W columns that has the launch to itself: where the tiles of
// two still leave a quarter of the SMs without one.  A tile is then half the work of a
// block (one round of its threads in most passes, 123 registers instead of 64 and
// spills).  An iteration of 64 x 1280 21.4 -> 14.5 us, 128 x 1792 26.5 -> 18.9, 222 x 2000
// 33 -> 29; a transform of 128 x 1715 11.7 -> 10.3 us.
inline bool mx_few_columns(int n, int W) { return n > 1024 && (W + 1) / 2 <= 111; }

// Whether the columns of a plain blur run in tiles of 32 rows instead of 128 (`tiles` of
// them, 32 columns each): where those leave SMs without a tile.  Columns of a blur with
// 19 taps, 32 rows and 128: 640 x 1024 (160 tiles) 6.4 and 6.6 us, 900 x 700 (174) 7.3 and
// 7.4, 1500 x 500 (188) 8.5 and 7.8, 1024 x 1024 (256) 8.1 and 6.9; 3 taps 5.2 and 5.3, 6.0 and
// 6.1, 7.1 and 6.5, 6.7 and 5.7.
inline bool vblur_small_tiles(int tiles) { return tiles < 6 * kSms / 5; }

// A thread of the random field makes 124 << shift numbers (kRandChunk) one after
// another, from a start that it reaches by matrix products.  Few numbers leave a
// short chain, many leave few products: us at shifts 0, 1, 2, 3 for 512 x 384 numbers
// 32, 43, 70, 113; 2048^2 56, 56, 84, 128; 6 Mi 75, 83, 85, 129; 8 Mi 103, 83, 88, 131; 12 Mi 141, 116, 148, 130;
// 4096^2 181, 157, 148, 137; 32 Mi 334, 293, 342, 313.  Shift 3 is the best of them only
// while its blocks of 128 threads are about one per SM.
inline int rand_chunk_shift(long n)
{
    if (n < 7000000) return 0;
    return n > 14000000 && n <= kSms * 128L * (124 << 3) ? 3 : 1;
}

}  // namespace imr
