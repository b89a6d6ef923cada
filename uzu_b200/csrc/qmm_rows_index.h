// Where a step of qmm_rows_kernel finds a feature's zero points. Plain C++: the kernel and a test on the host use the same function.
#pragma once
#include <cstdint>

namespace uzu {

struct QrZeroFetch {
    uint32_t offset, bytes, shift;      // a source on a 4-byte boundary, what of its word lies inside the array, bits in front of the step's zero points
};

// step_bytes: 4, or 2 with groups of 128. Rows are zp_stride bytes apart, an even number; where it is no multiple of four the array may end in the middle
// of the last word.
constexpr QrZeroFetch qr_zero_fetch(uint32_t row, uint32_t step, uint32_t n, uint32_t zp_stride, uint32_t step_bytes) {
    const uint32_t at = row * zp_stride + step * step_bytes, word = at & ~3u, left = n * zp_stride - word;
    return {word, left < 4u ? left : 4u, (at & 3u) * 8u};
}

}  // namespace uzu
