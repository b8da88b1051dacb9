// The Ewald terms of the FP64 pair kernel from a table of polynomials in s =
// (alpha r)^2.  With the Boys functions F_m(s) = integral_0^1 t^2m e^(-s t^2) dt
// and their complements C_m(s), the same integral from 1 to infinity,
//   force:  [erfc(alpha r) + 2 alpha r e^-s / sqrt(pi)] / (alpha r)^3
//             = 4/sqrt(pi) C_1(s) = s^(-3/2) - 4/sqrt(pi) F_1(s)
//   energy: erfc(alpha r) / (alpha r) = 2/sqrt(pi) C_0(s) = s^(-1/2) - 2/sqrt(pi) F_0(s)
// and dF_m/ds = -F_(m+1), dC_m/ds = -C_(m+1).  Row 0 covers s < 1/16 with the
// F form, which the kernel adds to the bare Coulomb term (of which it is a
// quarter at most, so hardly a digit cancels); all other rows hold the C form
// itself, so the term's rounding error is a share of the term, not of the bare
// one.  Rows are 1/128 of an octave up to s = 8 and 1/32 from there on, as far
// as the cutoffs of the context reach; each is a polynomial of degree 6 about
// its centre: the Taylor series to degree 13, its higher powers expressed by
// lower ones (Chebyshev economization), which leaves less than 1e-16 of the
// term.  Error of a single force term against long-precision values, in units
// of 1e-16, RMS over distances about 0.2, 0.5, 0.8 and 0.99 of a 1 nm cutoff:
// tolerance 5e-4 1.7, 2.3, 4.3, 4.0 (formed by erfc and exp: 2.6, 4.0, 8.4,
// 9.8; as a difference throughout: 2.2, 6.2, 60, 650); 1e-19: 2.7, 11, 28, 38
// (3.9, 16, 43, 53).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <cmath>
#include <mutex>
#include <vector>

namespace nxm {

constexpr int kEwaldRow = 8;     // doubles per row: coefficients of t^0..t^6 about the centre, the centre
constexpr int kEwaldOctave = 7;  // log2 of the rows per octave of s in [1/16, 8)
constexpr int kEwaldLinear = 1 + 7 * (1 << kEwaldOctave);  // first row from s = 8 on, 32 per unit

// Row of s (not checked against the table's end).
__host__ __device__ __forceinline__ int ewald_row(float s) {
    uint32_t b;
#ifdef __CUDA_ARCH__
    b = __float_as_uint(s);
#else
    memcpy(&b, &s, sizeof b);
#endif
    const int k = (int)(b >> (23 - kEwaldOctave)) - ((127 - 4) << kEwaldOctave) + 1;
    return s >= 8.0f ? kEwaldLinear + (int)((fminf(s, 4096.0f) - 8.0f) * 32.0f) : (k > 0 ? k : 0);
}

// The polynomial of a row (16-byte aligned) at r^2 alpha2.
__host__ __device__ __forceinline__ double ewald_poly(const double *row, double r2, double alpha2) {
    const double2 *c = reinterpret_cast<const double2 *>(row);
#ifdef __CUDA_ARCH__
    const double2 c67 = __ldg(c + 3), c45 = __ldg(c + 2), c23 = __ldg(c + 1), c01 = __ldg(c);
#else
    const double2 c67 = c[3], c45 = c[2], c23 = c[1], c01 = c[0];
#endif
    const double t = fma(r2, alpha2, -c67.y);
    double p = fma(c67.x, t, c45.y);
    p = fma(p, t, c45.x);
    p = fma(p, t, c23.y);
    p = fma(p, t, c23.x);
    p = fma(p, t, c01.y);
    return fma(p, t, c01.x);
}

// [erfc(alpha r) + 2 alpha r e^-s / sqrt(pi)] / r^3 (alphan: alpha^3) and
// erfc(alpha r) / r (alphan: alpha) from p, the polynomial of row `row` of the
// force's and of the energy's rows; `bare` is 1/r^3 and 1/r.
__host__ __device__ __forceinline__ double ewald_term(int row, double p, double alphan, double bare) {
    return fma(alphan, p, row == 0 ? bare : 0.0);
}

// The rows for s up to smax, force then energy, into `out`; returns the number
// of each.  Rows are made once per process.
inline int ewald_rows(double smax, std::vector<double> &out) {
    constexpr int N = 13, D = 6;
    static std::mutex mu;
    static std::vector<double> rows[2];
    static double low[N + 1][D + 1];  // u^n, n > D, on [-1, 1] by lower powers
    const int n = ewald_row((float)(smax * (1.0 + 1e-5))) + 1;
    std::lock_guard<std::mutex> lock(mu);
    if (rows[0].empty())
        for (int n0 = D + 1; n0 <= N; ++n0) {
            double b[N + 1] = {};
            b[n0] = 1.0;
            for (int k = n0; k > D; --k) {
                // b's power k by T_k / 2^(k-1) less its own lower powers
                double t0[N + 1] = {1.0}, t1[N + 1] = {0.0, 1.0};
                for (int m = 2; m <= k; ++m)
                    for (int c = N; c >= 0; --c) {
                        const double t2 = (c ? 2.0 * t1[c - 1] : 0.0) - t0[c];
                        t0[c] = t1[c];
                        t1[c] = t2;
                    }
                const double share = b[k] / t1[k];
                for (int c = 0; c <= k; ++c) b[c] -= share * t1[c];
            }
            for (int c = 0; c <= D; ++c) low[n0][c] = b[c];
        }
    const double sqrt_pi = 1.77245385090551602729;
    for (int k = (int)rows[0].size() / kEwaldRow; k < n; ++k) {
        // the row's range [s0, s0 + 2 h), its centre exact in FP64
        double s0, h;
        if (k == 0) {
            s0 = 0.0;
            h = 0x1p-5;
        } else if (k < kEwaldLinear) {
            const int e = ((k - 1) >> kEwaldOctave) - 4, m = (k - 1) & ((1 << kEwaldOctave) - 1);
            h = std::ldexp(1.0, e - kEwaldOctave - 1);
            s0 = std::ldexp(1.0, e) + 2.0 * h * m;
        } else {
            h = 0x1p-6;
            s0 = 8.0 + 2.0 * h * (k - kEwaldLinear);
        }
        const double s = s0 + h, ex = std::exp(-s);
        double B[N + 2];  // F_m or C_m at the centre
        if (k == 0) {
            // the series at the highest order, whose terms are all positive,
            // and downward from there
            constexpr int M = N + 1;
            double term = 1.0 / (2 * M + 1), sum = term;
            for (int j = 1; term > sum * 1e-18; ++j) {
                term *= 2.0 * s / (2 * M + 2 * j + 1);
                sum += term;
            }
            B[M] = ex * sum;
            for (int m = M - 1; m >= 0; --m) B[m] = (2.0 * s * B[m + 1] + ex) / (2 * m + 1);
        } else {
            // C_0 = sqrt(pi)/2 erfc(sqrt s) / sqrt s, the root's rounding put
            // right to first order; upward with positive terms only
            const double x = std::sqrt(s), dx = std::fma(-x, x, s) / (2.0 * x);
            B[0] = (0.5 * sqrt_pi * std::erfc(x) - ex * dx) / x * (1.0 - dx / x);
            for (int m = 0; m <= N; ++m) B[m + 1] = ((2 * m + 1) * B[m] + ex) / (2.0 * s);
        }
        for (int which = 0; which < 2; ++which) {
            // which 0: force (m = 1), 1: energy (m = 0); coefficients in u = t / h
            double a[N + 1], f = (which ? 2.0 : 4.0) / sqrt_pi * (k == 0 ? -1.0 : 1.0);
            for (int c = 0; c <= N; ++c) {
                a[c] = f * B[c + (which ? 0 : 1)];
                f *= -h / (c + 1);
            }
            for (int m = N; m > D; --m)
                for (int c = 0; c <= D; ++c) a[c] += a[m] * low[m][c];
            double hn = 1.0;
            for (int c = 0; c <= D; ++c, hn *= h) rows[which].push_back(a[c] / hn);
            rows[which].push_back(s);
        }
    }
    out.assign(rows[0].begin(), rows[0].begin() + (size_t)n * kEwaldRow);
    out.insert(out.end(), rows[1].begin(), rows[1].begin() + (size_t)n * kEwaldRow);
    return n;
}

}  // namespace nxm
