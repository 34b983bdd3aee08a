// Sine and cosine of the displacement (R6 of mp_device.cuh) and of its
// derivatives.  Only the rounded operations fadd ... ffma2 that mp_device.cuh
// defines before this file, so that the tests can run it on the host with
// their own.
#pragma once

#ifndef MP_TRIG_FN
#define MP_TRIG_FN __device__ __forceinline__
#endif

namespace mp {

// Cosine for the adjoint's derivatives: Cody-Waite reduction with pi/2 =
// P1 + P2 + P3 (three floats from the exact value of pi) and Taylor
// polynomials (degree 9 / 10) on |r| <= pi/4, with fused multiply-adds.
MP_TRIG_FN void sincos_reduced(float x, float& sr, float& cr, int& q) {
    float k = rintf(fmul(x, 0x1.45f306p-1f));
    float r = ffma(-k, 0x1.921fb6p+0f, x);
    r = ffma(-k, -0x1.777a5cp-25f, r);
    r = ffma(-k, -0x1.ee59dap-50f, r);
    float kq = fsub(k, fmul(4.0f, floorf(fmul(k, 0.25f))));
    q = (int)kq;
    float r2 = fmul(r, r);
    float ps = ffma(r2, 0x1.71de3ap-19f, -0x1.a01a02p-13f);
    ps = ffma(r2, ps, 0x1.111112p-7f);
    ps = ffma(r2, ps, -0x1.555556p-3f);
    sr = ffma(fmul(r, r2), ps, r);
    float pc = ffma(r2, -0x1.27e4fcp-22f, 0x1.a01a02p-16f);
    pc = ffma(r2, pc, -0x1.6c16c2p-10f);
    pc = ffma(r2, pc, 0x1.555556p-5f);
    pc = ffma(r2, pc, -0x1.0p-1f);
    cr = ffma(r2, pc, 1.0f);
}
// R6 native_sin: reduction by pi = PI1 + PI2 + PI3 (the pi/2 split doubled,
// exactly) to |r| <= pi/2, the odd Taylor polynomial of degree 13, the sign
// of (-1)^k; one polynomial instead of the two of sincos_reduced.
MP_TRIG_FN float mp_sinf(float x) {
    if (!isfinite(x)) return fsub(x, x);
    const float k = rintf(fmul(x, 0x1.45f306p-2f));
    float r = ffma(-k, 0x1.921fb6p+1f, x);
    r = ffma(-k, -0x1.777a5cp-24f, r);
    r = ffma(-k, -0x1.ee59dap-49f, r);
    const float r2 = fmul(r, r);
    float p = ffma(r2, 0x1.612462p-33f, -0x1.ae6456p-26f);
    p = ffma(r2, p, 0x1.71de3ap-19f);
    p = ffma(r2, p, -0x1.a01a02p-13f);
    p = ffma(r2, p, 0x1.111112p-7f);
    p = ffma(r2, p, -0x1.555556p-3f);
    const float sn = ffma(fmul(r, r2), p, r);
    const float odd = fsub(k, fmul(2.0f, floorf(fmul(k, 0.5f))));
    return odd != 0.0f ? -sn : sn;
}
MP_TRIG_FN float mp_cosf(float x) {
    if (!isfinite(x)) return fsub(x, x);
    float s, c;
    int q;
    sincos_reduced(x, s, c, q);
    q &= 3;
    return q == 0 ? c : q == 1 ? -s : q == 2 ? -c : s;
}

// mp_sinf for |x| < 2^22 pi, one value and a packed pair, bit for bit: k is
// rounded by adding and taking away 1.5 * 2^23 (round to nearest even, as
// rintf, with no conversion instruction), its parity is the sum's lowest bit,
// and k * -P equals -k * P.  x * (1 / pi) stays a scalar product: a packed
// one feeding the packed sum could be fused with it.
constexpr float kRintMagic = 12582912.0f;
MP_TRIG_FN float sin_small(float x) {
    const float km = fadd(fmul(x, 0x1.45f306p-2f), kRintMagic);
    const float k = fsub(km, kRintMagic);
    float r = ffma(k, -0x1.921fb6p+1f, x);
    r = ffma(k, 0x1.777a5cp-24f, r);
    r = ffma(k, 0x1.ee59dap-49f, r);
    const float r2 = fmul(r, r);
    float p = ffma(r2, 0x1.612462p-33f, -0x1.ae6456p-26f);
    p = ffma(r2, p, 0x1.71de3ap-19f);
    p = ffma(r2, p, -0x1.a01a02p-13f);
    p = ffma(r2, p, 0x1.111112p-7f);
    p = ffma(r2, p, -0x1.555556p-3f);
    const float sn = ffma(fmul(r, r2), p, r);
    return __uint_as_float(__float_as_uint(sn) ^ (__float_as_uint(km) << 31));
}
MP_TRIG_FN float2 sin2_small(float x, float y) {
    const float2 km = fadd2(make_float2(fmul(x, 0x1.45f306p-2f), fmul(y, 0x1.45f306p-2f)), dup2(kRintMagic));
    const float2 k = fadd2(km, dup2(-kRintMagic));
    float2 r = ffma2(k, dup2(-0x1.921fb6p+1f), make_float2(x, y));
    r = ffma2(k, dup2(0x1.777a5cp-24f), r);
    r = ffma2(k, dup2(0x1.ee59dap-49f), r);
    const float2 r2 = fmul2(r, r);
    float2 p = ffma2(r2, dup2(0x1.612462p-33f), dup2(-0x1.ae6456p-26f));
    p = ffma2(r2, p, dup2(0x1.71de3ap-19f));
    p = ffma2(r2, p, dup2(-0x1.a01a02p-13f));
    p = ffma2(r2, p, dup2(0x1.111112p-7f));
    p = ffma2(r2, p, dup2(-0x1.555556p-3f));
    const float2 sn = ffma2(fmul2(r, r2), p, r);
    return make_float2(__uint_as_float(__float_as_uint(sn.x) ^ (__float_as_uint(km.x) << 31)),
                       __uint_as_float(__float_as_uint(sn.y) ^ (__float_as_uint(km.y) << 31)));
}

// mp_cosf for |x| < 2^21 pi, one value and a pair, bit for bit, for the
// adjoint; the quadrant from the sum's lowest bits (the constant is a multiple
// of 4).  The one value has the two polynomials as the halves of one packed
// chain.  One even polynomial on sin_small's reduction (|r| <= pi/2) had a
// largest error of 1.5e-7 over [-44, 44] instead of 6.8e-8, an rms of 3.0e-8
// instead of 1.7e-8.  (backward() on the displaced 512x512 heightfield at
// 3840x2160: 0.640 ms with that, 0.696 with these one by one, 0.619 in pairs,
// the sines too.)
MP_TRIG_FN float cos_small(float x) {
    const float km = fadd(fmul(x, 0x1.45f306p-1f), kRintMagic);
    const float k = fsub(km, kRintMagic);
    float r = ffma(k, -0x1.921fb6p+0f, x);
    r = ffma(k, 0x1.777a5cp-25f, r);
    r = ffma(k, 0x1.ee59dap-50f, r);
    const float r2 = fmul(r, r);
    float2 p = make_float2(0x1.71de3ap-19f, ffma(r2, -0x1.27e4fcp-22f, 0x1.a01a02p-16f));
    p = ffma2(dup2(r2), p, make_float2(-0x1.a01a02p-13f, -0x1.6c16c2p-10f));
    p = ffma2(dup2(r2), p, make_float2(0x1.111112p-7f, 0x1.555556p-5f));
    p = ffma2(dup2(r2), p, make_float2(-0x1.555556p-3f, -0x1.0p-1f));
    const float2 sc = ffma2(make_float2(fmul(r, r2), r2), p, make_float2(r, 1.0f));
    // quadrants 0 to 3: c, -s, -c, s
    const unsigned q = __float_as_uint(km);
    return __uint_as_float(__float_as_uint(q & 1u ? sc.x : sc.y) ^ (((q + 1u) & 2u) << 30));
}

MP_TRIG_FN float2 cos2_small(float x, float y) {
    const float2 km = fadd2(make_float2(fmul(x, 0x1.45f306p-1f), fmul(y, 0x1.45f306p-1f)), dup2(kRintMagic));
    const float2 k = fadd2(km, dup2(-kRintMagic));
    float2 r = ffma2(k, dup2(-0x1.921fb6p+0f), make_float2(x, y));
    r = ffma2(k, dup2(0x1.777a5cp-25f), r);
    r = ffma2(k, dup2(0x1.ee59dap-50f), r);
    const float2 r2 = fmul2(r, r);
    float2 ps = ffma2(r2, dup2(0x1.71de3ap-19f), dup2(-0x1.a01a02p-13f));
    float2 pc = ffma2(r2, dup2(-0x1.27e4fcp-22f), dup2(0x1.a01a02p-16f));
    ps = ffma2(r2, ps, dup2(0x1.111112p-7f));
    pc = ffma2(r2, pc, dup2(-0x1.6c16c2p-10f));
    ps = ffma2(r2, ps, dup2(-0x1.555556p-3f));
    pc = ffma2(r2, pc, dup2(0x1.555556p-5f));
    const float2 s = ffma2(fmul2(r, r2), ps, r);
    pc = ffma2(r2, pc, dup2(-0x1.0p-1f));
    const float2 c = ffma2(r2, pc, dup2(1.0f));
    const unsigned qx = __float_as_uint(km.x), qy = __float_as_uint(km.y);
    return make_float2(__uint_as_float(__float_as_uint(qx & 1u ? s.x : c.x) ^ (((qx + 1u) & 2u) << 30)),
                       __uint_as_float(__float_as_uint(qy & 1u ? s.y : c.y) ^ (((qy + 1u) & 2u) << 30)));
}

}  // namespace mp
