// film.cuh -- mean and variance of the mean of a film value from its sums.
//
// mean = sum / count and var = (sumsq / count - mean^2) / (count - 1), rounded once from 64-bit
// arithmetic.  For an FP32 film of fewer than 2^24 samples the same values come from pairs of
// FP32 numbers (error-free products and differences: Dekker 1971, Knuth TAOCP 2, 4.2.2), which
// hold 48 bits: FP64 runs at a 64th of the FP32 rate here and its three divisions per value
// took 436 us of a 1080p film read-out, this form 32 us (bound by the film's bytes).  The mean
// is the correctly rounded quotient either way (53 >= 2 * 24 + 2 bits).  Sums whose products
// could overflow or lose bits to denormals take the 64-bit form.
#pragma once

#include "internal.h"

namespace salty {

struct FilmScale {
    double count;
    float n, inv;     // count and 1 / count (n = 0: always the 64-bit form)
    float fh, fl;     // 1 / (count - 1) as a pair
};

inline FilmScale film_scale(long long samples, bool fp64) {
    FilmScale s{(double)samples, 0.0f, 0.0f, 0.0f, 0.0f};
    if (fp64 || samples < 1 || samples >= (1ll << 24)) return s;
    s.n = (float)samples;
    s.inv = (float)(1.0 / (double)samples);
    if (samples > 1) {
        const double f = 1.0 / ((double)samples - 1.0);
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

__device__ __forceinline__ void film_value(float s, float q, const FilmScale& F, float& mean, float& var) {
    if (s == 0.0f && q == 0.0f) {
        mean = var = 0.0f;
        return;
    }
    mean = __fdiv_rn(s, F.n);
    const float p = mean * mean;
    if (!(F.n > 0.0f && q > 1e-25f && q < 1e30f && p > 1e-25f && p < 1e30f)) {
        film_value64((double)s, (double)q, F.count, mean, var);
        return;
    }
    const float ml = fmaf(-mean, F.n, s) * F.inv;   // mean + ml = s / n
    const float qh = __fdiv_rn(q, F.n);
    const float ql = fmaf(-qh, F.n, q) * F.inv;     // qh + ql = q / n
    const float pl = fmaf(2.0f * mean, ml, fmaf(mean, mean, -p));  // p + pl = (s / n)^2
    const float d = __fsub_rn(qh, p), b = __fsub_rn(d, qh);
    const float dl = __fadd_rn(__fsub_rn(__fsub_rn(qh, __fsub_rn(d, b)), __fadd_rn(p, b)), __fsub_rn(ql, pl));
    const float t = __fadd_rn(d, dl), tl = __fsub_rn(dl, __fsub_rn(t, d));
    const float v = __fmul_rn(t, F.fh);
    const float r = __fadd_rn(v, fmaf(t, F.fh, -v) + fmaf(t, F.fl, tl * F.fh));
    var = r > 0.0f ? r : 0.0f;
}

}  // namespace salty
