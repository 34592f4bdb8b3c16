// Sizes and places that outgrow 32 bits, for host and device.
#pragma once

#include <climits>
#include <cstdint>

#ifdef __CUDACC__
#define SEMO_HD __host__ __device__
#else
#define SEMO_HD
#endif

namespace semo {

// Slots of nslices slices of 32 rows that are all made `width` entries wide, or
// 0 when they are left as wide as their rows (`slots` in all): equal widths are
// taken from lo to hi, for at most an eighth of padding (more costs what the
// known place gains), and while a slot's place fits an int.
inline int64_t even_slots(int width, int lo, int hi, int64_t nslices, int64_t slots) {
    if (width < lo || width > hi) return 0;
    const int64_t even = 32 * (int64_t)width * nslices;
    return even <= slots + slots / 8 && even < INT_MAX ? even : 0;
}

// The row of a thread in a grid of `lanes` threads a row; rows times lanes may
// be above INT_MAX.
SEMO_HD inline int64_t row_of(unsigned block, unsigned threads, unsigned thread, int lanes) {
    return ((int64_t)block * threads + thread) / lanes;
}

}  // namespace semo
