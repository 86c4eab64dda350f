// row_copy.h - which rows of a frame come into shared memory in whole pieces.
//
// A strip's part of a row is copied in the 16-byte pieces that hold a byte of it.
// By the frame's first and last byte such a piece can reach up to 15 bytes past
// the frame, so the first and the last row, and every row of a frame whose rows
// are shorter than that, come in 4-byte words instead: nothing is read but the
// aligned words that hold the frame's bytes.  (A test by the addresses themselves,
// for every row, cost a frame 2 to 4%; this one at most 1%: float frames 59.9 -> 60.5 us
// at 1281x719, RGB24 frames of 3840x2160 218.5 either way.)
#pragma once

#ifdef __CUDACC__
#define WEMA_HD __host__ __device__ __forceinline__
#else
#define WEMA_HD static inline
#endif

namespace wema {

// rows 1 .. inner_rows of a frame of `rows` rows may be copied in whole pieces
WEMA_HD int inner_rows(int rows, int row_bytes) { return row_bytes >= 15 && rows > 2 ? rows - 2 : 0; }
WEMA_HD bool row_inner(int row, int inner) { return (unsigned)(row - 1) < (unsigned)inner; }

}  // namespace wema
