// Device-side RPC camera evaluation shared by the projection and camera-approximation
// kernels.  Two arithmetics:
//
//  * exact: FP64 in the reference's operation order (lib/rpc_model.py:52-62,160-168),
//    explicit round-to-nearest intrinsics so nothing is contracted into an FMA -- the
//    result is bit-identical to the numpy code;
//  * fast: GB300 runs FP64 at ~1/64 of the FP32 rate, so the fast form splits each FP64
//    input into a double-float (hi + lo floats) with integer operations, normalises and
//    evaluates the dominant constant+linear terms in double-float, the sixteen small
//    higher-order terms in plain FP32 (their magnitude bounds their rounding), and takes
//    the num/den ratio and the denormalisation in double-float.  |error| < 1e-4 px for
//    images up to 8192 px with WorldView-like coefficient magnitudes.
#pragma once

#include "common.cuh"

namespace vs {

// Per-camera constants of the fast form, prepared once per call.  The four polynomials
// travel as two (col, row) pairs through packed FP32x2 arithmetic: pair 0 = (colNum,
// rowNum), pair 1 = (colDen, rowDen).
struct RpcFast {
    df lat_off, lon_off, alt_off;       // offsets (double-float)
    df inv_lat, inv_lon, inv_alt;       // 1 / scale (double-float)
    float2 lin_hi[2][4], lin_lo[2][4];  // [pair][0..3] constant + linear coefficients
    float2 lin_nhi[2][4];               // -lin_hi (error terms of the products)
    float2 hot[2][16];                  // [pair][k-4] higher-order coefficients (FP32)
    float2 scale_hi, scale_lo, scale_nhi, off_hi, off_lo;   // (col, row) denormalisation
    float width, height;
};

// ---- exact FP64 (reference order) ------------------------------------------------------
__device__ __forceinline__ double dm(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double da(double a, double b) { return __dadd_rn(a, b); }

__device__ __forceinline__ double poly_exact(const double *c, double x, double y, double z) {
    double out = da(0.0, c[0]);
    out = da(out, da(da(dm(c[1], y), dm(c[2], x)), dm(c[3], z)));
    out = da(out, da(da(dm(dm(c[4], y), x), dm(dm(c[5], y), z)), dm(dm(c[6], x), z)));
    out = da(out, da(da(dm(dm(c[7], y), y), dm(dm(c[8], x), x)), dm(dm(c[9], z), z)));
    out = da(out, dm(dm(dm(c[10], x), y), z));
    out = da(out, dm(dm(dm(c[11], y), y), y));
    out = da(out, da(da(dm(dm(dm(c[12], y), x), x), dm(dm(dm(c[13], y), z), z)), dm(dm(dm(c[14], y), y), x)));
    out = da(out, dm(dm(dm(c[15], x), x), x));
    out = da(out, da(da(dm(dm(dm(c[16], x), z), z), dm(dm(dm(c[17], y), y), z)), dm(dm(dm(c[18], x), x), z)));
    out = da(out, dm(dm(dm(c[19], z), z), z));
    return out;
}

// ---- exact FP64 with the products on the integer pipes -----------------------------------
// A polynomial is 45 products and 19 sums, and GB300's FP64 pipe does 1.65 of either per clock
// and SM (measured; 32-bit integer work ~60, mul.wide.u32 22), so the FP64 form above is
// bound by its products.  A product rounded to nearest even is integer arithmetic: the 53-bit
// significands' 106-bit product, one normalising shift, and the round-up carried into the
// exponent -- 4 wide multiplies and ~17 logic operations, 2.8 products per clock and SM,
// beside the sums that stay on the FP64 pipe.  Same bits as __dmul_rn as long as every operand is
// zero or of moderate exponent, so that no partial product leaves the normal range (``moderate``,
// asked of each factor and coefficient).  The four polynomials of a point: 1.92 -> 5.02
// Gpoints/s; the projection of 214,221 points by 12 cameras 1672 -> 647 us (with the
// divisions of the normalisation as below).

// A factor of products: significand (hi has 21 bits), exponent word less the bias, and a mask
// that makes the products of a zero zero (their sign does not matter: a sum that starts
// from +0 never becomes -0).
struct Factor {
    unsigned hi, lo, ew, mask;
};
// A coefficient: significand, sign and exponent word, mask as above.
struct __align__(16) RpcCoef {
    unsigned hi, lo, ew, mask;
};

// Zero, or an exponent within 2^+-160: a product of four such numbers stays normal.
__device__ __forceinline__ bool moderate(double v) {
    const unsigned h = static_cast<unsigned>(__double2hiint(v)), l = static_cast<unsigned>(__double2loint(v));
    return ((h >> 20) & 0x7ffu) - (1023u - 160u) <= 320u || ((h << 1) | l) == 0u;
}
__device__ __forceinline__ unsigned zero_mask(double v) {
    const unsigned h = static_cast<unsigned>(__double2hiint(v)), l = static_cast<unsigned>(__double2loint(v));
    return ((h << 1) | l) == 0u ? 0u : ~0u;
}

__device__ __forceinline__ Factor factor_of(double v) {
    const unsigned h = static_cast<unsigned>(__double2hiint(v));
    return {(h & 0xfffffu) | 0x100000u, static_cast<unsigned>(__double2loint(v)), (h & 0xfff00000u) - (1024u << 20),
            zero_mask(v)};
}

__device__ __forceinline__ RpcCoef coef_of(double v) {
    const unsigned h = static_cast<unsigned>(__double2hiint(v));
    return {(h & 0xfffffu) | 0x100000u, static_cast<unsigned>(__double2loint(v)), h & 0xfff00000u, zero_mask(v)};
}

// (rh, rl) = the double (ahi, alo, aew) * b, rounded to nearest even.  The significands'
// product has 105 or 106 bits: a left shift by 12 or 11 leaves the 53 kept bits in (hh, hl)
// and the next 32 in lh.  Bits below those only matter as "not zero" (in `up`): adding
// 0x7fffffff + (odd or not zero) to lh carries exactly when the rest is above one half, or one
// half below an odd significand.
__device__ __forceinline__ void mul_bits(unsigned ahi, unsigned alo, unsigned aew, const Factor &b, unsigned &rh,
                                         unsigned &rl) {
    const unsigned long long t0 = static_cast<unsigned long long>(alo) * b.lo;
    unsigned long long mid = static_cast<unsigned long long>(alo) * b.hi;      // < 2^53
    mid += static_cast<unsigned long long>(ahi) * b.lo;
    mid += t0 >> 32;
    const unsigned long long top = static_cast<unsigned long long>(ahi) * b.hi + (mid >> 32);
    unsigned hh = static_cast<unsigned>(top >> 32), hl = static_cast<unsigned>(top), lh = static_cast<unsigned>(mid);
    const unsigned ll = static_cast<unsigned>(t0);
    const unsigned two = hh >> 9;                    // 1 when the product of the significands is >= 2
    const unsigned e = aew + b.ew + (two << 20);
    hh = __funnelshift_l(hl, hh, 12u - two);
    hl = __funnelshift_l(lh, hl, 12u - two);
    lh = __funnelshift_l(ll, lh, 12u - two);
    const unsigned up = (hl | min(ll, 1u)) & 1u;
    asm("{\n\t.reg .u32 t;\n\t"
        "add.u32 t, %3, 0x7fffffff;\n\t"
        "add.cc.u32 t, %2, t;\n\t"
        "addc.cc.u32 %0, %4, 0;\n\t"
        "addc.u32 %1, %5, %6;\n\t}"
        : "=r"(rl), "=r"(rh)
        : "r"(lh), "r"(up), "r"(hl), "r"(hh), "r"(e));
}

// A product on its way through its factors.
struct Prod {
    unsigned h, l, mask;
};
__device__ __forceinline__ Prod operator*(const RpcCoef &c, const Factor &f) {
    Prod p;
    p.mask = c.mask & f.mask;
    mul_bits(c.hi, c.lo, c.ew, f, p.h, p.l);
    return p;
}
__device__ __forceinline__ Prod operator*(const Prod &a, const Factor &f) {
    Prod p;
    p.mask = a.mask & f.mask;
    mul_bits((a.h & 0xfffffu) | 0x100000u, a.l, a.h & 0xfff00000u, f, p.h, p.l);
    return p;
}
__device__ __forceinline__ double value(const Prod &p) {
    return __hiloint2double(static_cast<int>(p.h & p.mask), static_cast<int>(p.l & p.mask));
}
// The constant term, da(0.0, c) of the reference: +0 for either zero.
__device__ __forceinline__ double value(const RpcCoef &c) {
    return __hiloint2double(static_cast<int>((c.ew | (c.hi & 0xfffffu)) & c.mask), static_cast<int>(c.lo & c.mask));
}

// poly_exact over coefficients and factors that are moderate: the same bits.
__device__ __forceinline__ double poly_factors(const RpcCoef *c, const Factor &x, const Factor &y, const Factor &z) {
    double out = value(c[0]);
    out = da(out, da(da(value(c[1] * y), value(c[2] * x)), value(c[3] * z)));
    out = da(out, da(da(value(c[4] * y * x), value(c[5] * y * z)), value(c[6] * x * z)));
    out = da(out, da(da(value(c[7] * y * y), value(c[8] * x * x)), value(c[9] * z * z)));
    out = da(out, value(c[10] * x * y * z));
    out = da(out, value(c[11] * y * y * y));
    out = da(out, da(da(value(c[12] * y * x * x), value(c[13] * y * z * z)), value(c[14] * y * y * x)));
    out = da(out, value(c[15] * x * x * x));
    out = da(out, da(da(value(c[16] * x * z * z), value(c[17] * y * y * z)), value(c[18] * x * x * z)));
    out = da(out, value(c[19] * z * z * z));
    return out;
}

// v / d, rounded to nearest even, for a divisor known in advance: with the reciprocal as a
// double-word (hi = RN(1/d), lo = 1/d - hi to 53 bits), q = RN(v hi + RN(v lo)) is a
// double next to v / d on either side (Brisebarre, Muller, Raina, "Accelerating correctly rounded
// floating-point division when the divisor is known in advance", IEEE TC 53(8), 2004), the
// residual v - d q is exact, and RN(q + r hi) is the rounded quotient (Markstein, IBM J.
// R&D 34(1), 1990).  4 FP64 operations against about 10 of a division.  v and d moderate.
struct Divisor {
    double d, hi, lo;
};
__device__ __forceinline__ Divisor divisor_of(double d) {
    const double hi = __drcp_rn(d);
    return {d, hi, __dmul_rn(hi, __fma_rn(-d, hi, 1.0))};
}
__device__ __forceinline__ double div_known(double v, const Divisor &d) {
    const double q = __fma_rn(v, d.hi, __dmul_rn(v, d.lo));
    return __fma_rn(__fma_rn(-d.d, q, v), d.hi, q);
}

// One camera of the exact projection in shared memory: the camera, its four polynomials'
// coefficients (in the camera's order: row_num, row_den, col_num, col_den), the divisors of
// the normalisation, and whether all of these are moderate.
struct RpcExact {
    VsRpcCamera cam;
    RpcCoef coef[80];
    Divisor lat, lon, alt;
    int moderate;
};

__device__ __forceinline__ void load_exact(const VsRpcCamera *__restrict__ src, RpcExact &s) {
    const double *d = reinterpret_cast<const double *>(src);
    double *cam = reinterpret_cast<double *>(&s.cam);
    if (threadIdx.x == 0) s.moderate = 1;
    __syncthreads();
    for (int i = threadIdx.x; i < static_cast<int>(sizeof(VsRpcCamera) / 8); i += blockDim.x) {
        const double v = d[i];
        cam[i] = v;
        if (i >= 10 && i < 90) s.coef[i - 10] = coef_of(v);
        const bool scale = i == 5 || i == 7 || i == 9;
        if (scale) (i == 5 ? s.lat : (i == 7 ? s.lon : s.alt)) = divisor_of(v);
        if ((scale && v == 0.0) || ((scale || (i >= 10 && i < 90)) && !moderate(v))) s.moderate = 0;
    }
    __syncthreads();
}

// (v - offset) / scale.
__device__ __forceinline__ double normalise_exact(bool known, double v, double off, const Divisor &d) {
    const double a = __dsub_rn(v, off);
    return known && moderate(a) ? div_known(a, d) : __ddiv_rn(a, d.d);
}

// The four polynomials at (lat, lon, alt) = (x, y, z), normalised, in the camera's order.
__device__ __forceinline__ void polys_exact(const RpcExact &s, double x, double y, double z, double (&p)[4]) {
    if (s.moderate && moderate(x) && moderate(y) && moderate(z)) {
        const Factor fx = factor_of(x), fy = factor_of(y), fz = factor_of(z);
        // one polynomial at a time: four in flight would not raise the rate, and cost registers
        auto store = [&](int q, double v) {
            p[0] = q == 0 ? v : p[0];
            p[1] = q == 1 ? v : p[1];
            p[2] = q == 2 ? v : p[2];
            p[3] = q == 3 ? v : p[3];
        };
#pragma unroll 1
        for (int q = 0; q < 4; ++q) store(q, poly_factors(s.coef + 20 * q, fx, fy, fz));
    } else {
        p[0] = poly_exact(s.cam.row_num, x, y, z);
        p[1] = poly_exact(s.cam.row_den, x, y, z);
        p[2] = poly_exact(s.cam.col_num, x, y, z);
        p[3] = poly_exact(s.cam.col_den, x, y, z);
    }
}

__device__ __forceinline__ void project_exact(const RpcExact &s, double lat, double lon, double alt, double &col,
                                              double &row) {
    const VsRpcCamera &cam = s.cam;
    const bool known = s.moderate != 0;
    const double c_lon = normalise_exact(known, lon, cam.lon_off, s.lon);
    const double c_lat = normalise_exact(known, lat, cam.lat_off, s.lat);
    const double c_alt = normalise_exact(known, alt, cam.alt_off, s.alt);
    double p[4] = {0.0, 0.0, 0.0, 0.0};
    polys_exact(s, c_lat, c_lon, c_alt, p);
    col = da(dm(__ddiv_rn(p[2], p[3]), cam.col_scale), cam.col_off);
    row = da(dm(__ddiv_rn(p[0], p[1]), cam.row_scale), cam.row_off);
}

// ---- fast (double-float) ------------------------------------------------------------------
// Splits an FP64 value into hi + lo floats without FP64 arithmetic: hi keeps the top 24
// significant bits (truncated from the bit pattern, so the remainder is exact), lo is the
// remaining 29 bits converted to a float (one rounding) and scaled by their power of two.
// Magnitudes outside 2^+-100 (zero, tiny, huge, inf, NaN) become the nearest float with
// lo = 0.  The integer conversion is one instruction (measured faster here than the
// two-halves float trick it replaced, the fit 2.69 -> 2.64 ms).
__device__ __forceinline__ df split_double(double v) {
    const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(v));
    const int e = static_cast<int>((b >> 52) & 0x7ff);
    if (e < 1023 - 100 || e > 1023 + 100) return {f64_to_f32(v), 0.0f};
    const unsigned sign = static_cast<unsigned>(b >> 32) & 0x80000000u;
    const unsigned mant_hi = static_cast<unsigned>((b >> 29) & 0x7fffffu);   // top 23 fraction bits
    const float hi = __uint_as_float(sign | (static_cast<unsigned>(e - 1023 + 127) << 23) | mant_hi);
    const unsigned rest = static_cast<unsigned>(b & 0x1fffffffu);            // low 29 fraction bits
    // value of the low bits: rest * 2^(e - 1075); 2^(e-1075) = 2^(e-1023) * 2^-52
    const float scale = __uint_as_float(static_cast<unsigned>(e - 1023 - 52 + 127) << 23);
    float lo = __uint2float_rn(rest) * scale;
    lo = sign ? -lo : lo;
    return {hi, lo};
}

// constant + three linear terms in double-float, plus the FP32 higher-order sum, for the
// two polynomials of a pair at once (same operations per lane as the scalar form: exact
// products of the high parts with their cross terms in the low word, the TwoSum chain of
// constant, linear terms and higher-order sum)
__device__ __forceinline__ df2 poly_fast2(const float2 (&hi)[4], const float2 (&lo)[4], const float2 (&nhi)[4],
                                          const float2 (&hot)[16], df x, df y, df z, const float (&m)[16]) {
    const float2 Y = f2s(y.hi), X = f2s(x.hi), Z = f2s(z.hi);
    // two_prod(c, v): -fl(c v) = fl((-c) v) from the negated coefficients
    const df2 p1 = {__fmul2_rn(hi[1], Y), __ffma2_rn(hi[1], Y, __fmul2_rn(nhi[1], Y))};
    const df2 p2 = {__fmul2_rn(hi[2], X), __ffma2_rn(hi[2], X, __fmul2_rn(nhi[2], X))};
    const df2 p3 = {__fmul2_rn(hi[3], Z), __ffma2_rn(hi[3], Z, __fmul2_rn(nhi[3], Z))};
    float2 low = __fadd2_rn(__fadd2_rn(__fadd2_rn(lo[0], p1.lo), p2.lo), p3.lo);
    low = __ffma2_rn(hi[1], f2s(y.lo), __ffma2_rn(lo[1], Y, low));
    low = __ffma2_rn(hi[2], f2s(x.lo), __ffma2_rn(lo[2], X, low));
    low = __ffma2_rn(hi[3], f2s(z.lo), __ffma2_rn(lo[3], Z, low));
    float2 h = f2s(0.0f);
#pragma unroll
    for (int k = 0; k < 16; ++k) h = __ffma2_rn(hot[k], f2s(m[k]), h);
    df2 s = two_sum2(hi[0], p1.hi);
    low = __fadd2_rn(low, s.lo);
    s = two_sum2(s.hi, p2.hi);
    low = __fadd2_rn(low, s.lo);
    s = two_sum2(s.hi, p3.hi);
    low = __fadd2_rn(low, s.lo);
    s = two_sum2(s.hi, h);
    low = __fadd2_rn(low, s.lo);
    return fast_two_sum2(s.hi, low);
}

// monomials 4..19 of the RPC order from the high parts of the normalised coordinates
__device__ __forceinline__ void monomials(float x, float y, float z, float (&m)[16]) {
    const float yx = y * x, yz = y * z, xz = x * z, yy = y * y, xx = x * x, zz = z * z;
    m[0] = yx; m[1] = yz; m[2] = xz; m[3] = yy; m[4] = xx; m[5] = zz;
    m[6] = yx * z;       // xyz
    m[7] = yy * y;       // y^3
    m[8] = y * xx;       // y x^2
    m[9] = y * zz;       // y z^2
    m[10] = yy * x;      // y^2 x
    m[11] = xx * x;      // x^3
    m[12] = x * zz;      // x z^2
    m[13] = yy * z;      // y^2 z
    m[14] = xx * z;      // x^2 z
    m[15] = zz * z;      // z^3
}

// (v - off) * inv: the difference's error is ~2^-48 of |v| (a few 1e-13 degrees), far below
// what the 1e-4 px bound allows after the scale.
__device__ __forceinline__ df normalise(df v, df off, df inv) {
    return df_mul(df_add_ops(v, {-off.hi, -off.lo}), inv);
}

// (col, row) as double-floats for one point given as split lat/lon/alt: the numerator
// pair and the denominator pair, then both quotients and denormalisations as one pair.
__device__ __forceinline__ void project_fast(const RpcFast &c, df lat, df lon, df alt, df &col, df &row) {
    const df x = normalise(lat, c.lat_off, c.inv_lat);
    const df y = normalise(lon, c.lon_off, c.inv_lon);
    const df z = normalise(alt, c.alt_off, c.inv_alt);
    float m[16];
    monomials(x.hi, y.hi, z.hi, m);
    const df2 num = poly_fast2(c.lin_hi[0], c.lin_lo[0], c.lin_nhi[0], c.hot[0], x, y, z, m);
    const df2 den = poly_fast2(c.lin_hi[1], c.lin_lo[1], c.lin_nhi[1], c.hot[1], x, y, z, m);
    // quotients through a Newton-refined reciprocal (relative error < 2^-43)
    const df2 r = df_recip2(den);
    const df2 q = df_mul2(num, r, sub2(f2s(0.0f), r.hi));
    const df2 v = df_add_ops2(df_mul2(q, {c.scale_hi, c.scale_lo}, c.scale_nhi), {c.off_hi, c.off_lo});
    col = {v.hi.x, v.lo.x};
    row = {v.hi.y, v.lo.y};
}

// df < float bound, for the in-image mask (col >= 0, col < width)
__device__ __forceinline__ bool df_lt(df a, float b) { return a.hi < b || (a.hi == b && a.lo < 0.0f); }
__device__ __forceinline__ bool df_ge0(df a) { return a.hi > 0.0f || (a.hi == 0.0f && a.lo >= 0.0f); }

// Fills an RpcFast from a camera, the block's threads sharing its 49 conversions (one thread
// alone spent 10 us on their FP64 instructions).  Ends with a barrier.
__device__ __forceinline__ void prepare_fast(const VsRpcCamera &cam, RpcFast &f) {
    const double *polys[2][2] = {{cam.col_num, cam.row_num}, {cam.col_den, cam.row_den}};
    for (int t = threadIdx.x; t < 49; t += blockDim.x) {
        if (t < 3) {
            const df v = df_from_double(t == 0 ? cam.lat_off : (t == 1 ? cam.lon_off : cam.alt_off));
            (t == 0 ? f.lat_off : (t == 1 ? f.lon_off : f.alt_off)) = v;
        } else if (t < 6) {
            const df v = df_from_double(1.0 / (t == 3 ? cam.lat_scale : (t == 4 ? cam.lon_scale : cam.alt_scale)));
            (t == 3 ? f.inv_lat : (t == 4 ? f.inv_lon : f.inv_alt)) = v;
        } else if (t < 14) {
            const int p = (t - 6) >> 2, k = (t - 6) & 3;
            const df a = df_from_double(polys[p][0][k]), b = df_from_double(polys[p][1][k]);
            f.lin_hi[p][k] = make_float2(a.hi, b.hi);
            f.lin_lo[p][k] = make_float2(a.lo, b.lo);
            f.lin_nhi[p][k] = make_float2(-a.hi, -b.hi);
        } else if (t < 46) {
            const int p = (t - 14) >> 4, k = (t - 14) & 15;
            f.hot[p][k] = make_float2(static_cast<float>(polys[p][0][k + 4]), static_cast<float>(polys[p][1][k + 4]));
        } else if (t < 48) {
            const df c = df_from_double(t == 46 ? cam.col_scale : cam.col_off);
            const df r = df_from_double(t == 46 ? cam.row_scale : cam.row_off);
            if (t == 46) {
                f.scale_hi = make_float2(c.hi, r.hi);
                f.scale_lo = make_float2(c.lo, r.lo);
                f.scale_nhi = make_float2(-c.hi, -r.hi);
            } else {
                f.off_hi = make_float2(c.hi, r.hi);
                f.off_lo = make_float2(c.lo, r.lo);
            }
        } else {
            f.width = static_cast<float>(cam.width);
            f.height = static_cast<float>(cam.height);
        }
    }
    __syncthreads();
}

}  // namespace vs
