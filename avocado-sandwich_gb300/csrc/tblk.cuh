// The buffer of the panel's 16 x 16 T blocks, and the counters of the full-T trailing
// update (tiles of 128 and 256), which take its place once the T build has read it.
// Host arithmetic only.
#pragma once

#include <stddef.h>
#include <stdint.h>

namespace avs {

// Elements of the buffer for a matrix of order n: nt + 1 tiles, whatever part of a panel
// one launch has.
constexpr size_t tblk_elems(int64_t n, int b) { return (size_t)(n / b + 1) * (size_t)(b / 16) * 256; }

// The update's split: columns of a strip and rows of W handed on at once.
constexpr int upd_strip(int elem_bytes, bool narrow) { return elem_bytes == 8 ? (narrow ? 16 : 32) : 64; }
constexpr int upd_row_block(int elem_bytes, int b) { return elem_bytes == 8 && b == 256 ? 16 : 32; }
// A ticket and a counter per row block of each strip: at most ncols + 1 ints, in a
// buffer of 16 (ncols + 2 b) elements.
constexpr int64_t upd_strips(int64_t ncols, int strip) { return (ncols + strip - 1) / strip; }
constexpr int64_t upd_counters(int64_t ncols, int b, int elem_bytes, int strip) {
    return 1 + upd_strips(ncols, strip) * (b / upd_row_block(elem_bytes, b));
}

}  // namespace avs
