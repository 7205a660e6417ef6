// How a launch's blocks share a list of segments. Plain C++, so that the
// arithmetic is checked on the host for lists of every length, empty ones among
// them.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define PB_HOST_DEVICE __host__ __device__
#else
#define PB_HOST_DEVICE
#endif

namespace pb {

// Segments begin, begin + 1, ... of block y of ny: ``chunk`` at a time, from
// ``step`` further on each time, up to ``end``.
struct SegSlice {
    int64_t begin, end, step, chunk;
};

// A contiguous slice of ``live`` segments a block, or (``dealt``) equal chunks
// dealt out over the blocks in turn; at most ``most`` segments a chunk. chunk and
// step are at least 1 whatever the list, so a block's loop always ends; an empty
// list gives every block an empty slice.
PB_HOST_DEVICE inline SegSlice seg_slice(int64_t live, int64_t y, int64_t ny, int64_t most, bool dealt) {
    SegSlice s{0, 0, most, most};
    if (live <= 0) return s;
    const int64_t per = (live + ny - 1) / ny;
    if (dealt) {
        const int64_t rounds = (per + most - 1) / most;
        s.chunk = (per + rounds - 1) / rounds;
        s.step = s.chunk * ny;
        s.begin = s.chunk * y < live ? s.chunk * y : live;
        s.end = live;
    } else {
        s.begin = per * y < live ? per * y : live;
        s.end = s.begin + per < live ? s.begin + per : live;
    }
    return s;
}

}  // namespace pb
