// decode_schedule.h -- order of the tiled posterior decoding (decode.cu): which
// row blocks' cells tile (I, J = I + D) reads, and which flags its CTA waits
// for before it reads them.  Plain C++, so that the order can be walked on the
// host as well.
#pragma once

#ifdef __CUDACC__
#define MESSI_SCHEDULE_FN __host__ __device__ __forceinline__
#else
#define MESSI_SCHEDULE_FN inline
#endif

namespace messi {

// flags[block] >= diagonals: the tiles (block, block) .. (block, block +
// diagonals - 1) are written.  diagonals <= 0: nothing to wait for.
struct DecodeWait {
    int block, diagonals;
};

// Row blocks [first, J) of the split points that are taken before the late
// wait, and what orders them: with row block I + 3 done up to diagonal D - 3,
// its tile (I + 3, J) is written, and as that tile waited for row block I + 4
// up to D - 4, and so on, so is every (R, J) with R >= I + 3.  (The late wait of
// the row block's previous tile says nothing of column J: it proves row block
// I + k up to diagonal D - 1 - k, column J - 1.)
MESSI_SCHEDULE_FN int decode_early_first(int I) { return I + 3; }

MESSI_SCHEDULE_FN DecodeWait decode_early_wait(int I, int D)
{
    return D >= 4 ? DecodeWait{I + 3, D - 2} : DecodeWait{I, 0};  // D < 4: there are none
}

// Before the rest: the two row blocks next to the tile's own, its column
// block's diagonal tile and the neighbours of its cells.
MESSI_SCHEDULE_FN DecodeWait decode_late_wait(int I, int D) { return DecodeWait{I + 1, D}; }

}  // namespace messi
