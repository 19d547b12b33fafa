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
// `cols_resident`, `rows_resident`: blocks that run at the same time.
inline bool fft_rows_start_early(int cols, int cols_resident, int rows, int rows_resident)
{
    return rows <= 111 || cols >= 2 * kSms || rows > rows_resident || (rows <= kSms && cols_resident > kSms);
}

// Whether the columns of a plain transform run in narrow tiles (4 columns) instead
// of the wide ones (`wide_tiles` of them; 16 columns up to H = 512, 8 at 1024):
// where the wide tiles leave half of the SMs without one.  Whole transform, wide ->
// narrow: 256 x 256 6.2 -> 5.2 us (16 wide tiles), 512 x 1024 10.5 -> 8.9 (64); beyond
// that narrow tiles only make the strides shorter: 2048 x 512 13.0 -> 13.9 (128),
// 2048 x 1024 23.8 -> 25.0 (256), 4096 x 64 7.7 -> 8.0.
inline bool fft_narrow_columns(int wide_tiles) { return 2 * wide_tiles < kSms; }

}  // namespace imr
