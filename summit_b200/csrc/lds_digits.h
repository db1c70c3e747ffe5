// The four balanced base-128 digits of a 28-bit value and their rounding, in
// 32-bit arithmetic that may wrap (unsigned throughout).  Free of CUDA types, so
// that the CPU tests compile it as it is.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define LDS_HD __host__ __device__ __forceinline__
#else
#define LDS_HD inline
#endif

namespace lds {
namespace umma {

// The balanced base-128 digits of a 28-bit sketch value R = d0 128^3 + d1 128^2
// + d2 128 + d3 (d1..d3 in [-63, 64]) as the bytes of one word, d3 lowest.
// U = R + 63 (128^2 + 128 + 1) has the digits' 7-bit fields (plus 63) in place;
// two multiply-adds spread them to bytes (top field first by 2, then the upper
// field of each half by 1), and adding 65 and flipping the top bit subtracts 63
// from each of the low three bytes without a borrow.
LDS_HD uint32_t digits_word(int32_t R) {
    const uint32_t U = (uint32_t)R + 63u * (16384u + 128u + 1u);
    const uint32_t y = U + 3u * (U & 0xFFFFC000u);
    return (y + (y & 0xFF803F80u) + 0x00414141u) ^ 0x00808080u;
}

// The shift that narrow_round applies: right by r (0..14) to the nearest even.
struct NarrowShift {
    int32_t r;      // right shift of the low digits' part
    int32_t up;     // 14 - r: left shift of the high digits' part
    int32_t half;   // half an ulp less one
    int32_t odd;    // parity mask
};
LDS_HD NarrowShift narrow_shift(int32_t r) {
    return NarrowShift{r, 14 - r, r > 0 ? (1 << ((r - 1) & 15)) - 1 : 0, r > 0 ? 1 : 0};
}

// rint(T 2^-r), ties to even, for T = ((t0 128 + t1) 128 + t2) 128 + t3 whose
// result fits 32 bits and whose low part L = 128 t2 + t3 is below 2^31 - 2^14 in
// magnitude: with H = 128 t0 + t1 it is H 2^(14-r) + rint(L 2^-r), the tie parity
// taken from the whole value.  H's multiple may wrap, and with it the sum's terms,
// hence unsigned; the sum modulo 2^32 is the result.
LDS_HD int32_t narrow_round(int32_t t0, int32_t t1, int32_t t2, int32_t t3, NarrowShift sh) {
    const int32_t L = t2 * 128 + t3;
    const uint32_t A = ((uint32_t)t0 * 128u + (uint32_t)t1) << sh.up;
    const uint32_t odd = (A + (uint32_t)(L >> sh.r)) & (uint32_t)sh.odd;
    return (int32_t)(A + (uint32_t)((L + sh.half + (int32_t)odd) >> sh.r));
}

}  // namespace umma
}  // namespace lds
