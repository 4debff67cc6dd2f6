// film.cuh -- mean and variance of the mean of a film value from its sums.
//
// mean = sum / count and var = (sumsq / count - mean^2) / (count - 1) = (count sumsq - sum^2) /
// (count^2 (count - 1)).  For an FP32 film of fewer than 2^24 samples the numerator is exact:
// both products are 48 bits, held as pairs of FP32 numbers, and their difference keeps every
// rounding error as a further term (error-free products and differences: Dekker 1971, Knuth
// TAOCP 2, 4.2.2).  So the variance is the exact one rounded once, whatever cancels: 0.50 units
// in the last place at every spread, where FP64 quotients reach 0.60 at a variance of 2^-23 of
// the squared mean and 4 at 2^-24.  FP64 runs at a 64th of the FP32 rate here and its three
// divisions per value took 436 us of a 1080p film read-out, this form 32 us (bound by the film's
// bytes).  The mean is the correctly rounded quotient either way (53 >= 2 * 24 + 2 bits).  Sums
// whose products could overflow or lose bits to denormals take the 64-bit form.
#pragma once

#include "internal.h"

namespace salty {

struct FilmScale {
    double count;
    float n;          // count (0: always the 64-bit form)
    float fh, fl;     // 1 / (count^2 (count - 1)) as a pair (0 for one sample)
};

inline FilmScale film_scale(long long samples, bool fp64) {
    FilmScale s{(double)samples, 0.0f, 0.0f, 0.0f};
    if (fp64 || samples < 1 || samples >= (1ll << 24)) return s;
    s.n = (float)samples;
    if (samples > 1) {
        const double n = (double)samples, f = 1.0 / (n * n * (n - 1.0));
        s.fh = (float)f;
        s.fl = (float)(f - (double)s.fh);
    }
    return s;
}

__device__ __forceinline__ void film_value64(double s, double q, double count, float& mean, float& var) {
    const double m = count > 0 ? s / count : 0.0;
    mean = (float)m;
    const double v = count > 1 ? (q / count - m * m) * count / (count - 1.0) / count : 0.0;
    var = (float)(v > 0 ? v : 0.0);
}

// a + b and its rounding error (Knuth's TwoSum).
__device__ __forceinline__ float two_sum(float a, float b, float& err) {
    const float t = __fadd_rn(a, b), z = __fsub_rn(t, a);
    err = __fadd_rn(__fsub_rn(a, __fsub_rn(t, z)), __fsub_rn(b, z));
    return t;
}

__device__ __forceinline__ void film_value(float s, float q, const FilmScale& F, float& mean, float& var) {
    if (s == 0.0f && q == 0.0f) {
        mean = var = 0.0f;
        return;
    }
    const float ph = __fmul_rn(F.n, q), pl = fmaf(F.n, q, -ph);  // count sumsq
    const float sh = __fmul_rn(s, s), sl = fmaf(s, s, -sh);      // sum^2
    if (!(F.n > 0.0f && ph > 1e-25f && ph < 1e37f && sh > 1e-25f && sh < 1e37f)) {
        film_value64((double)s, (double)q, F.count, mean, var);
        return;
    }
    mean = __fdiv_rn(s, F.n);
    var = 0.0f;
    if (F.fh == 0.0f) return;
    float e, le, tl;
    const float d = two_sum(ph, -sh, e), l = two_sum(pl, -sl, le), t = two_sum(d, l, tl);
    const float rest = __fadd_rn(tl, __fadd_rn(e, le));
    const float hi = __fadd_rn(t, rest), lo = __fsub_rn(rest, __fsub_rn(hi, t));
    if (!(hi > 0.0f)) return;
    const float v = __fmul_rn(hi, F.fh);
    if (v < 0x1p-100f) {  // the correction's terms would be denormal
        film_value64((double)s, (double)q, F.count, mean, var);
        return;
    }
    var = __fadd_rn(v, fmaf(hi, F.fh, -v) + fmaf(hi, F.fl, lo * F.fh));
}

}  // namespace salty
