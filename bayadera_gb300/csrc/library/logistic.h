// Bayesian logistic regression: data rows (x_1..x_F, y) with y in {0, 1}, F = dim;
// hyperparameter h0 = prior sd of every coefficient.
// log density = sum_n [y_n eta_n - softplus(eta_n)] - |beta|^2 / (2 h0^2),
// eta_n = x_n . beta, softplus(e) = max(e, 0) + log(1 + exp(-|e|)); log(1 + t) for
// t = exp(-|e|) in (0, 1] has an absolute rounding error below 2^-24 (fast-math exp and
// log are single MUFU operations; log1pf is not).
#include <stdint.h>
extern "C" {
inline REAL logistic_softplus(const REAL e) { return fmaxf(e, 0.0f) + logf(1.0f + expf(-fabsf(e))); }
inline REAL logistic_logpdf(const uint32_t data_len, const uint32_t hyper_len,
                            const REAL* params, const uint32_t dim, const REAL* beta) {
    const uint32_t row = dim + 1, n = data_len / row;
    REAL res = 0.0f;
    for (uint32_t i = 0; i < n; ++i) {
        const REAL* r = params + (uint64_t)i * row;
        REAL eta = 0.0f;
        for (uint32_t f = 0; f < dim; ++f) eta = fmaf(r[f], beta[f], eta);
        res += fmaf(r[dim], eta, -logistic_softplus(eta));
    }
    const REAL sd = params[data_len];
    REAL pr = 0.0f;
    for (uint32_t f = 0; f < dim; ++f) pr = fmaf(beta[f], beta[f], pr);
    return res - pr / (2.0f * sd * sd);
}
// GEMM form: A = the data rows' features, aux = y.
inline void logistic_prep(const REAL* hyper, const uint32_t hyper_len, const uint32_t dim,
                          const REAL* beta, REAL* prep) {}
inline REAL logistic_term(const REAL eta, const REAL* aux, const uint64_t row, const REAL* beta,
                          const REAL* prep) {
    return fmaf(aux[0], eta, -logistic_softplus(eta));
}
// 16 rows' terms at once, aux = their y.  The rows' log(1 + exp(-|eta|)) are one logarithm
// of a running product of 1 + exp(-|eta|), in (1, 2] each: carry holds the mantissas, in
// [1, 2), of the even and the odd rows' products and their exponents' sum (an integer's
// bits), and logistic_term_16_end gives the product's -log as hi + lo.  A multiplication's relative
// rounding error, 2^-24 at most, is one of the sum; a fast-math logarithm a row has an
// absolute one of about 2^-23.  The exponential's argument is raised by 4e-8: fast math's
// exp2 comes out low by that much of an octave on average, which no longer cancels against the
// logarithms' mean error.  Relative RMS errors against 64 bits over 1,048,576 x 64, 100,000 x 20,
// 50,007 x 128, 400,000 x 200 and 10,000 x 3 (rows x features): a logarithm a row 5.2, 4.5, 6.9,
// 10.7 and 2.5e-8; this without the raise 5.5, 4.5, 7.4, 11.2 and 2.8e-8, with it 5.2, 4.4,
// 6.9, 10.2 and 2.5e-8.
// y eta - max(eta, 0) is taken row by row, exact for y of 0 or 1: summed apart, rows that are
// classified right leave the rounding error of their |eta| where any other row is not (normal
// eta of scale 100, 2 % of the labels flipped: 8.2e-6 RMS a batch of 16 rows, row by row 1.1e-6).
inline REAL logistic_exp_neg_abs(const REAL eta) {
    return exp2f(fmaf(fabsf(eta), -1.44269504f, 4.0e-8f));
}
inline void logistic_term_16_init(REAL* carry) {
    carry[0] = carry[1] = 1.0f;
    carry[2] = __int_as_float(0);
}
inline REAL logistic_term_16(const REAL* eta, const REAL* aux, const uint64_t row, const REAL* beta,
                             const REAL* prep, REAL* carry) {
    bay_f2 p = bay_f2_of(carry[0], carry[1]), s = bay_f2_of(0.0f, 0.0f);
#pragma unroll
    for (int i = 0; i < 16; i += 2) {
        const bay_f2 t = bay_f2_of(logistic_exp_neg_abs(eta[i]), logistic_exp_neg_abs(eta[i + 1]));
        p = bay_f2_fma(p, t, p);
        // y eta - max(eta, 0), exact for y of 0 or 1
        s = bay_f2_add(s, bay_f2_fma(bay_f2_of(aux[i], aux[i + 1]), bay_f2_of(eta[i], eta[i + 1]),
                                     bay_f2_of(fminf(-eta[i], 0.0f), fminf(-eta[i + 1], 0.0f))));
    }
    const int b0 = __float_as_int(bay_f2_x(p)), b1 = __float_as_int(bay_f2_y(p));
    carry[2] = __int_as_float(__float_as_int(carry[2]) + (b0 >> 23) + (b1 >> 23) - 254);
    carry[0] = __int_as_float((b0 & 0x007fffff) | 0x3f800000);
    carry[1] = __int_as_float((b1 & 0x007fffff) | 0x3f800000);
    return bay_f2_x(s) + bay_f2_y(s);
}
inline REAL logistic_term_16_end(const REAL* carry, REAL* lo) {
    const REAL e = (REAL)__float_as_int(carry[2]);
    const REAL h = __fmul_rn(e, 0.693147182f);               // ln 2 = 0.693147182 - 1.90465e-9
    *lo = -(fmaf(e, -1.90465430e-9f, fmaf(e, 0.693147182f, -h)) + logf(carry[0] * carry[1]));
    return -h;
}
inline REAL logistic_walker(const uint64_t rows, const REAL* hyper, const uint32_t hyper_len,
                            const uint32_t dim, const REAL* beta) {
    REAL pr = 0.0f;
    for (uint32_t f = 0; f < dim; ++f) pr = fmaf(beta[f], beta[f], pr);
    return -pr / (2.0f * hyper[0] * hyper[0]);
}
}
// Streamed tensor-core form: the epilogue's instruction issue bounds it; an exponential, a
// logarithm and the scalar sums a row took 8,192 walkers x 1,048,653 rows of 64 features 4,160
// us, these 2,680 to 2,770 (the split products alone 1,730 at the measured rate).
#if BAY_GEMM_AUX <= 1          // a row's y and nothing else
#define logistic_term_16_carry 3
#endif
