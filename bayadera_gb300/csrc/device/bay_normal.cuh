// bay_normal.cuh -- the Box-Muller pair of the normal walker init, in pairs of floats with the
// FP64 evaluation where they leave the rounding open.
//
// The init is defined by an FP64 formula rounded to fp32: x = mean + sd r cos(t) and
// mean + sd r sin(t), r = sqrt(-2 log u1), t = 6.283185307179586 u0.  FP64 issue is 1/64 of
// fp32 on this part and the pair takes some 95 FP64 operations.  Here r, cos and sin are
// evaluated as unevaluated sums of two floats (r to about 2^-41, cos and sin to 2^-44; series from
// the functions' definitions, exact sums and products after Knuth and Dekker), and the rounding
// to fp32 is accepted where every value within the error bound rounds alike (Ziv's test);
// where not, some 2^-14 of the elements, the caller takes the FP64 formula.  The results are
// the FP64 formula's, bit for bit.
#ifndef BAY_NORMAL_CUH
#define BAY_NORMAL_CUH

struct bay_df {
    float h, l;
};
// a + b for |a| >= |b| or a = 0
__device__ __forceinline__ bay_df bay_df_fast(float a, float b) {
    const float s = __fadd_rn(a, b);
    return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ bay_df bay_df_sum(float a, float b) {
    const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
    return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t))};
}
__device__ __forceinline__ bay_df bay_df_mul(bay_df a, bay_df b) {
    const float p = __fmul_rn(a.h, b.h);
    float e = __fmaf_rn(a.h, b.h, -p);
    e = __fmaf_rn(a.h, b.l, e);
    e = __fmaf_rn(a.l, b.h, e);
    return bay_df_fast(p, e);
}
// c + p for |c| >= |p|
__device__ __forceinline__ bay_df bay_df_add(bay_df c, bay_df p) {
    const bay_df s = bay_df_fast(c.h, p.h);
    return bay_df_fast(s.h, __fadd_rn(s.l, __fadd_rn(c.l, p.l)));
}

// log u, 0 < u < 1 (normal): u = m 2^e, m in [sqrt 1/2, sqrt 2), log m = 2 atanh s,
// s = (m - 1) / (m + 1), |s| < 0.172, by the atanh series to s^19.
__device__ __forceinline__ bay_df bay_df_log(float u) {
    const int b = __float_as_int(u);
    int e = (b >> 23) - 127;
    float m = __int_as_float((b & 0x007fffff) | 0x3f800000);
    if (m > 1.41421354f) {
        m = __fmul_rn(m, 0.5f);
        e += 1;
    }
    const float f = __fsub_rn(m, 1.0f);
    const bay_df d = bay_df_fast(2.0f, f);                    // m + 1
    const float q = __fdividef(f, d.h);
    const float r = __fmaf_rn(-q, d.l, __fmaf_rn(-q, d.h, f));
    const bay_df s = bay_df_fast(q, __fdividef(r, d.h));
    const bay_df w = bay_df_mul(s, s);
    float t = __fmaf_rn(w.h, 1.0f / 19.0f, 1.0f / 17.0f);
    t = __fmaf_rn(w.h, t, 1.0f / 15.0f);
    t = __fmaf_rn(w.h, t, 1.0f / 13.0f);
    t = __fmaf_rn(w.h, t, 1.0f / 11.0f);
    t = __fmaf_rn(w.h, t, 1.0f / 9.0f);
    t = __fmaf_rn(w.h, t, 1.0f / 7.0f);
    constexpr float fifth = 0.2f, third = 1.0f / 3.0f;
    const bay_df q1 = bay_df_add({fifth, (float)(0.2 - (double)fifth)}, {__fmul_rn(w.h, t), 0.0f});
    const bay_df q0 = bay_df_add({third, (float)(1.0 / 3.0 - (double)third)}, bay_df_mul(w, q1));
    bay_df g = bay_df_add(s, bay_df_mul(bay_df_mul(s, w), q0));
    g.h = __fadd_rn(g.h, g.h);
    g.l = __fadd_rn(g.l, g.l);
    if (e == 0) return g;
    // e ln 2 with ln 2 in three parts, the first of 16 bits (its product is exact)
    constexpr double ln2 = 0.693147180559945309417;
    constexpr float h = 0.693145751953125f, mid = (float)(ln2 - (double)h);
    constexpr float low = (float)(ln2 - (double)h - (double)mid);
    const float fe = (float)e;
    const float pm = __fmul_rn(fe, mid), pe = __fmaf_rn(fe, mid, -pm);
    const bay_df s1 = bay_df_sum(__fmul_rn(fe, h), g.h);
    const bay_df s2 = bay_df_sum(pm, g.l);
    const bay_df s3 = bay_df_sum(s1.h, s2.h);
    return bay_df_fast(s3.h, __fadd_rn(__fadd_rn(s1.l, s3.l), __fadd_rn(s2.l, __fmaf_rn(fe, low, pe))));
}

// sqrt(-2 log u)
__device__ __forceinline__ bay_df bay_df_radius(float u) {
    const bay_df g = bay_df_log(u);
    const float vh = __fmul_rn(-2.0f, g.h), vl = __fmul_rn(-2.0f, g.l);
    const float r = __fmul_rn(vh, rsqrtf(vh));
    const float rem = __fadd_rn(__fmaf_rn(-r, r, vh), vl);
    return bay_df_fast(r, __fdividef(rem, __fadd_rn(r, r)));
}

// cos and sin of 2 pi u, 0 <= u <= 1: u = k / 4 + y exactly, |y| <= 1/8, Taylor series at
// 2 pi y, |2 pi y| <= pi / 4.
__device__ __forceinline__ void bay_df_circle(float u, bay_df& c, bay_df& s) {
    const float k = rintf(__fmul_rn(4.0f, u));
    const float y = __fmaf_rn(k, -0.25f, u);
    constexpr double pi2 = 6.283185307179586476925;
    constexpr float ph = (float)pi2, pl = (float)(pi2 - (double)ph);
    const float p = __fmul_rn(y, ph);
    const bay_df a = bay_df_fast(p, __fmaf_rn(y, pl, __fmaf_rn(y, ph, -p)));
    const bay_df w = bay_df_mul(a, a);
    constexpr double s3 = -1.0 / 6.0, s5 = 1.0 / 120.0, s7 = -1.0 / 5040.0;
    constexpr double c4 = 1.0 / 24.0, c6 = -1.0 / 720.0, c8 = 1.0 / 40320.0;
    float t = __fmaf_rn(w.h, (float)(-1.0 / 1307674368000.0), (float)(1.0 / 6227020800.0));
    t = __fmaf_rn(w.h, t, (float)(-1.0 / 39916800.0));
    t = __fmaf_rn(w.h, t, (float)(1.0 / 362880.0));
    bay_df q = bay_df_add({(float)s7, (float)(s7 - (double)(float)s7)}, {__fmul_rn(w.h, t), 0.0f});
    q = bay_df_add({(float)s5, (float)(s5 - (double)(float)s5)}, bay_df_mul(w, q));
    q = bay_df_add({(float)s3, (float)(s3 - (double)(float)s3)}, bay_df_mul(w, q));
    const bay_df sn = bay_df_add(a, bay_df_mul(bay_df_mul(a, w), q));
    t = __fmaf_rn(w.h, (float)(1.0 / 20922789888000.0), (float)(-1.0 / 87178291200.0));
    t = __fmaf_rn(w.h, t, (float)(1.0 / 479001600.0));
    t = __fmaf_rn(w.h, t, (float)(-1.0 / 3628800.0));
    q = bay_df_add({(float)c8, (float)(c8 - (double)(float)c8)}, {__fmul_rn(w.h, t), 0.0f});
    q = bay_df_add({(float)c6, (float)(c6 - (double)(float)c6)}, bay_df_mul(w, q));
    q = bay_df_add({(float)c4, (float)(c4 - (double)(float)c4)}, bay_df_mul(w, q));
    q = bay_df_add({-0.5f, 0.0f}, bay_df_mul(w, q));
    const bay_df cs = bay_df_add({1.0f, 0.0f}, bay_df_mul(w, q));
    const int kk = (int)k & 3;                                // quadrant
    c = (kk & 1) ? sn : cs;
    s = (kk & 1) ? cs : sn;
    if (kk == 1 || kk == 2) {
        c.h = -c.h;
        c.l = -c.l;
    }
    if (kk >= 2) {
        s.h = -s.h;
        s.l = -s.l;
    }
}

// mean + sd r g rounded to fp32 into x; false where the bound leaves the rounding open.  The
// bound: 2^-39 of the product (r and g), the FP64 formula's own 2^-49 of sd r (its angle is
// rounded), 2^-46 of the sum.
__device__ __forceinline__ bool bay_df_normal(float mean, float sd, bay_df r, bay_df g, float* x) {
    const bay_df z = bay_df_mul(r, g);
    const float p = __fmul_rn(sd, z.h);
    const bay_df q = bay_df_fast(p, __fmaf_rn(sd, z.l, __fmaf_rn(sd, z.h, -p)));
    const bay_df a = bay_df_sum(mean, q.h);
    const bay_df v = bay_df_fast(a.h, __fadd_rn(a.l, q.l));
    const float err = __fmaf_rn(fabsf(q.h), 1.8189894e-12f,
                                __fmaf_rn(fabsf(__fmul_rn(sd, r.h)), 1.7763568e-15f,
                                          __fmul_rn(fabsf(v.h), 1.4210855e-14f)));
    const float up = __fadd_rn(v.h, __fadd_rn(v.l, err)), down = __fadd_rn(v.h, __fsub_rn(v.l, err));
    *x = up;
    return up == down && fabsf(v.h) >= 1e-20f && fabsf(v.h) <= 1e30f;
}

#endif
