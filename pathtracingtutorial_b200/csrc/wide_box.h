// wide_box.h -- the 8-bit boxes of the four-wide tree: a node's grid on one
// axis and the codes of its children's planes (layout and argument in wide.h).
// Host and device give the same bits: the roundings are spelled out.
#pragma once

#include "pt_internal.h"

namespace ptb {

// a + b rounded down / up.
PT_HD float add_rd(float a, float b) {
#if defined(__CUDA_ARCH__)
    return __fadd_rd(a, b);
#else
    // hi + lo is the exact sum (two-sum in double)
    const double x = a, y = b, hi = x + y, t = hi - x, lo = (x - (hi - t)) + (y - t);
    const float s = static_cast<float>(hi);
    const double d = static_cast<double>(s) - hi;
    return d > 0.0 || (d == 0.0 && lo < 0.0) ? nextafterf(s, -FLT_MAX) : s;
#endif
}
PT_HD float add_ru(float a, float b) { return -add_rd(-a, -b); }

// D(code) of wide.h.
PT_HD float wide_decode(uint32_t code) { return __uint_as_float_hd(0x43000000u | (code << 16)); }

PT_HD float wide_scale(uint32_t exponent) { return __uint_as_float_hd(exponent << 23); }

// Grid of a node on one axis: the planes base + D(code) * scale from code 0 to
// 255 hold [mn, mx].  False when none was found (not for |mn|, |mx| <= 1e30:
// from 382 scale >= 2 (mx - mn) on, and 382 scale >= 5 ulp(max(|mn|, |mx|)),
// the grid reaches mx although rounding puts base up to an ulp below
// mn - 128 scale; both hold after two steps).  The second start matters for
// boxes with no or hardly any thickness on the axis -- a wall, a floor -- at a
// coordinate other than 0.
PT_HD bool wide_frame(float mn, float mx, float& base, uint32_t& exponent) {
    const float ext = add_ru(mx, -mn), most = fmaxf(fabsf(mn), fabsf(mx));
    int e = -100;
    if (ext > 0.0f) e = ilogbf(ext / 382.0f);
    if (most > 0.0f) {
        const int thin = ilogbf(most) - 31;
        if (e < thin) e = thin;
    }
    e = e < -100 ? -100 : (e > 100 ? 100 : e);
    for (int k = 0; k < 4; ++k, ++e) {
        exponent = static_cast<uint32_t>(e + 127);
        const float s = wide_scale(exponent);
        base = add_rd(mn, -128.0f * s);
        if (add_rd(510.0f * s, base) >= mx) return true;   // (510 s is exact)
    }
    return false;
}

// Largest code whose plane is at or below v / smallest at or above v, for v in
// the grid's interval.
PT_HD uint32_t wide_code_lo(float v, float base, float s) {
    const float x = fminf((v - base) / s, 512.0f);
    int c = x < 256.0f ? static_cast<int>(floorf(x)) - 128 : static_cast<int>(floorf(0.5f * x));
    c = c + 1 < 0 ? 0 : (c + 1 > 255 ? 255 : c + 1);
    while (c > 0 && add_ru(wide_decode(static_cast<uint32_t>(c)) * s, base) > v) --c;
    return static_cast<uint32_t>(c);
}
PT_HD uint32_t wide_code_hi(float v, float base, float s) {
    const float x = fminf((v - base) / s, 512.0f);
    int c = x <= 255.0f ? static_cast<int>(ceilf(x)) - 128 : static_cast<int>(ceilf(0.5f * x));
    c = c - 1 < 0 ? 0 : (c - 1 > 255 ? 255 : c - 1);
    while (c < 255 && add_rd(wide_decode(static_cast<uint32_t>(c)) * s, base) < v) ++c;
    return static_cast<uint32_t>(c);
}

}  // namespace ptb
