// Column tiles of rows that are copied by the aligned 16-byte vectors which cover them (seg_ragged_kernel).  Plain
// integer rules, in a header that a host compiler takes as well: tests walk them over every width and row begin.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define CGNN_COVER_FN __host__ __device__
#else
#define CGNN_COVER_FN
#endif

namespace cgnn {

// Columns of a tile: what `lpr` aligned vectors hold wherever a row begins.  With 4-byte units that is one column more than
// (lpr - 1) * 4, which would give every lane of a four-lane group a fourth element for it (width 1: 20.5 us a pass
// against 22.2).
CGNN_COVER_FN constexpr int ragged_tile(int lpr, int unit) { return unit == 4 ? (lpr - 1) * 4 : lpr * 4 - 2; }

// Whether the whole cover of the tile at column col0 may be copied: it holds up to lpr * 4 columns of the row (all of them
// when the row begins on a 16-byte boundary), and no byte behind the row is read.
CGNN_COVER_FN constexpr bool ragged_whole_cover(int lpr, int64_t width, int64_t col0) { return col0 + lpr * 4 <= width; }

}  // namespace cgnn
