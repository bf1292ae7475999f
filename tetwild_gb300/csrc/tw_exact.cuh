// tw_exact.cuh -- correctly rounded binary64 results with fewer binary64
// instructions (included by tw_device.cuh inside namespace tw).
//
// This GPU issues one binary64 warp instruction per 17 cycles and SM, 64 times
// less than binary32 or integer ones.  Where a binary64 operation only adds a
// small correction to a value, fl(y + c) with |c| below some million units of
// y's last place, the correction is needed to a few digits, not 53 bits: it is
// evaluated in binary32 in units of y's last place, rounded to a whole number
// and added to y's bits.  The result is that of the binary64 operation unless
// the correction lies within its binary32 error of a half unit, or the sum
// meets a power of two (where the unit changes); then ok = false and the
// caller does the binary64 operations.
#pragma once

__device__ __forceinline__ int exponent_field(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }

// A positive or negative normal number as binary32, truncated (relative error
// below 2^-22), with the exponent field set to 127: its significand in [1, 2).
__device__ __forceinline__ float significand32(double x) {
    const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
    return __uint_as_float(0x3f800000u | ((hi & 0xfffffu) << 3) | (lo >> 29));
}

// fl(|y| + (g + lo) units of y's last place), with y's sign; the error of
// g + lo is at most err (lo: what g's own rounding left, for large g).
__device__ __forceinline__ double add_units(double y, float g, float lo, float err, bool& ok) {
    const float k = rintf(g);
    const long long u = __double_as_longlong(y);
    const long long r = u + (long long)__float2int_rn(k);
    // the same exponent (and sign), neither a power of two, the rounding certain
    ok = ok && fabsf(g) < 4e6f && fabsf((g - k) + lo) < 0.5f - err &&
         ((u ^ r) & 0x7ff0000000000000LL) == 0 && (u & 0x000fffffffffffffLL) != 0 &&
         (r & 0x000fffffffffffffLL) != 0;
    return __longlong_as_double(r);
}

// Reciprocal of a normal d to about 2^-44 by one Newton step from a binary32
// seed on the significand; good: the exponents leave room for the residuals.
__device__ __forceinline__ double recip_seeded(double d, bool& good) {
    const int e = exponent_field(d);
    good = e > 523 && e < 1523;   // 2^-500 < |d| < 2^500
    const uint32_t s = __float_as_uint(__fdividef(1.0f, significand32(d)));   // in (1/2, 1]
    const uint32_t ef = (s >> 23) + 896u - (uint32_t)(e - 1023);
    const uint32_t hi = ((uint32_t)__double2hiint(d) & 0x80000000u) | (ef << 20) | ((s & 0x7fffffu) >> 3);
    const double r0 = __hiloint2double((int)hi, (int)(s << 29));
    return fma(r0, fma(-d, r0, 1.0), r0);
}

// c / d rounded to nearest, from r = recip_seeded(d): the quotient c r and its
// residual c - d (c r) (one fma, as in Markstein's "Computation of elementary
// functions on the IBM RISC System/6000 processor", 1990, sec. 3), whose
// quotient by d is a correction of at most 2^10 units.  Out of range, or when
// it cannot tell, the division itself.
static __device__ __noinline__ double div_ieee(double c, double d) { return c / d; }
__device__ __forceinline__ double div_seeded(double c, double d, double r, bool good) {
    const double q = c * r;
    const double rem = fma(-d, q, c);
    const int ec = exponent_field(c), eq = exponent_field(q), er = exponent_field(rem);
    bool ok = good && ec > 323 && ec < 1723;
    // rem r / unit(q): significands in binary32, the powers of two apart
    const int e = (er - 1023) + (exponent_field(r) - 1023) - (eq - 1023) + 52;   // 2^e
    const bool zero = er == 0;   // an exact quotient (rem is 0, or far below any unit)
    ok = ok && (zero || (e > -60 && e < 20));
    const uint32_t sgn = ((uint32_t)__double2hiint(rem) ^ (uint32_t)__double2hiint(r) ^
                          (uint32_t)__double2hiint(q)) & 0x80000000u;
    const float mag = significand32(rem) * significand32(r) *
                      __uint_as_float((uint32_t)(127 + max(-60, min(e, 20))) << 23);
    const float g = zero ? 0.0f : __uint_as_float(__float_as_uint(mag) | sgn);
    const double out = add_units(q, g, 0.0f, fmaf(fabsf(g), 1e-6f, 1e-6f), ok);
    return ok ? out : div_ieee(c, d);
}
