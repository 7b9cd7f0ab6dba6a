// kg_log.cuh — the logarithms of a pass over frequency nodes, by table: the
// library's log is 30 FP64 instructions, node_log 9.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#include <cuda_runtime.h>

namespace kg {

// 2^e for e = -LOG_BIAS .. LOG_EXPS - LOG_BIAS - 1: eps = 1e-8 is 2^-26.6, so a d
// (eps .. 1 + eps) and a ratio of two (5e-9 .. 2e8) lie inside.
constexpr int LOG_CELLS = 128, LOG_EXPS = 64, LOG_BIAS = 32;
struct LogTable {
    double2 cell[LOG_CELLS];   // {c, -log c}
    double exp2[LOG_EXPS];     // (e - LOG_BIAS) log 2
};

inline void fill_log_table(LogTable& T) {
    for (int i = 0; i < LOG_CELLS; i++) {
        const double c = 1.0 / (1.0 + (i + 0.5) / LOG_CELLS);
        T.cell[i] = make_double2(c, -std::log(c));
    }
    for (int i = 0; i < LOG_EXPS; i++) T.exp2[i] = (i - LOG_BIAS) * 0.69314718055994530942;
}

// log d for 2^-32 <= d < 2^32 (Tang, ACM TOMS 16, 1990): d = 2^e m, c the
// reciprocal of the middle of m's 1/128 interval, log d = e log 2 - log c +
// log1p(m c - 1), the last by its series (|m c - 1| < 2^-8: the first term left
// out is below 3e-18).
__host__ __device__ __forceinline__ double node_log(double d, const LogTable& T) {
#ifdef __CUDA_ARCH__
    const int hi = __double2hiint(d);
    const double m = __hiloint2double((hi & 0x000FFFFF) | 0x3FF00000, __double2loint(d));
#else
    uint64_t bits, one;
    std::memcpy(&bits, &d, 8);
    const int hi = (int)(bits >> 32);
    one = (bits & 0x000FFFFFFFFFFFFFull) | 0x3FF0000000000000ull;
    double m;
    std::memcpy(&m, &one, 8);
#endif
    const double2 c = T.cell[(hi >> 13) & (LOG_CELLS - 1)];
    const double r = fma(m, c.x, -1.0);
    double s = fma(r, -1.0 / 6.0, 0.2);
    s = fma(r, s, -0.25);
    s = fma(r, s, 1.0 / 3.0);
    s = fma(r, s, -0.5);
    s = fma(r * r, s, r);
    return (T.exp2[((hi >> 20) - 1023 + LOG_BIAS) & (LOG_EXPS - 1)] + c.y) + s;
}

// log(d / (d - delta)) = -log(1 - z), z = delta / d: the series for |z| <= 1/64
// (the first term left out is below 1e-15 of the sum), else the table.
__host__ __device__ __forceinline__ double node_neg_log1m(double z, const LogTable& T) {
    if (fabs(z) <= 0.015625) {
        double s = fma(z, 0.125, 1.0 / 7.0);
        s = fma(z, s, 1.0 / 6.0);
        s = fma(z, s, 0.2);
        s = fma(z, s, 0.25);
        s = fma(z, s, 1.0 / 3.0);
        s = fma(z, s, 0.5);
        s = fma(z, s, 1.0);
        return z * s;
    }
    return -node_log(1.0 - z, T);
}

}  // namespace kg
