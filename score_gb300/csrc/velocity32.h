// The FP32 velocity factor (float)((m p) f_geo) without FP64 arithmetic.
//
// FP64 runs at 1/64 of the FP32 rate here: two multiplications and a conversion a slot were what the fill of a
// front that refreshes its velocities every step (recovery) waited for.  The product is formed as a sum of two
// FP32 numbers instead, whose error is below 2^-42.6 of it (operands cut to 46 bits, products of low parts left out,
// roundings of the low part), the roundings of the FP64 product included.  If it rounds to the same FP32
// number 2^-40 above and below, that number is the FP64 result's rounding; if not (one slot in
// 2^16), or far outside the usual magnitudes, the caller computes in FP64.  A recovering 384^3 domain took 51.1 us a step, now
// 48.2; a heated 120^3 one 31.1 and 30.8.  Plain C++: the same bits on host and device.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define SCORE_HD __host__ __device__ __forceinline__
#else
#define SCORE_HD inline
#endif

namespace score {

SCORE_HD float float_of(uint32_t b) {
    float f;
    memcpy(&f, &b, 4);
    return f;
}
// positive double within 2^-90 .. 2^90
SCORE_HD bool split_range(uint64_t b) { return (uint32_t)(b >> 32) - (933u << 20) < (180u << 20); }
// its first 24 bits and the next 23
SCORE_HD void split_bits(uint64_t b, float& h, float& l) {
    const uint32_t hb = (uint32_t)(b >> 29) - (896u << 23), e = (hb & 0x7F800000u) - (23u << 23);
    h = float_of(hb);
    l = float_of(e | (((uint32_t)b << 3) >> 9)) - float_of(e);
}
// m, p: bits of the mobility and the driving force; code: infector code (shape factor 1, .7957 or .6494)
SCORE_HD bool velocity32(uint64_t m, uint64_t p, uint32_t code, float& v) {
    constexpr uint32_t kFace = 1u << 4 | 1u << 10 | 1u << 12 | 1u << 13 | 1u << 15 | 1u << 21 | 1u << 26;
    constexpr uint32_t kCorner = 1u << 0 | 1u << 2 | 1u << 6 | 1u << 8 | 1u << 17 | 1u << 19 | 1u << 23 | 1u << 25;
    constexpr float kEdgeHi = (float)0.7957, kEdgeLo = (float)(0.7957 - (double)kEdgeHi);
    constexpr float kCornerHi = (float)0.6494, kCornerLo = (float)(0.6494 - (double)kCornerHi);
    if (!split_range(m) || !split_range(p)) return false;
    const bool face = (kFace >> code) & 1u, corner = (kCorner >> code) & 1u;
    const float sh = face ? 1.0f : corner ? kCornerHi : kEdgeHi, sl = face ? 0.0f : corner ? kCornerLo : kEdgeLo;
    float mh, ml, ph, pl;
    split_bits(m, mh, ml);
    split_bits(p, ph, pl);
    const float h1 = mh * ph;
    if (!(h1 > 1e-24f && h1 < 1e24f)) return false;  // the low parts stay normal numbers
    float l1 = fmaf(mh, ph, -h1);
    l1 = fmaf(mh, pl, l1);
    l1 = fmaf(ml, ph, l1);
    const float h2 = h1 * sh;
    float l2 = fmaf(h1, sh, -h2);
    l2 = fmaf(h1, sl, l2);
    l2 = fmaf(l1, sh, l2);
    const float d = h2 * 9.0949470177292824e-13f;  // 2^-40
    const float up = h2 + (l2 + d);
    v = h2 + (l2 - d);
    return up == v;
}

}  // namespace score
