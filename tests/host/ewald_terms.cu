// Host-side check of the FP64 Ewald terms (compiled and run by
// tests/test_ewald_terms_host.py, no GPU): force and energy term of one pair
// from the table of nxm_ewald64.cuh against long double, at distances from
// 0.02 nm to the cutoff and across the table's seams.
//
// Largest error allowed, in units of 2^-53 of the term: alpha^2 is rounded
// once, which the term's slope turns into up to s + 3/2; alpha^3, the product
// with it and the polynomial's last step round once each; the row's leading
// coefficient is within 3, its truncation within 1, and in the first row the
// bare term's three roundings count 4/3: 9 + 1.1 s.  In the mean over a range
// the error may not pass that of the same terms formed by erfc and exp (a half
// more for the scatter of two samples).
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "../../nexusmd_gb300/csrc/nxm_ewald64.cuh"

using namespace nxm;

int main() {
    bool ok = true;
    const double ulp = std::ldexp(1.0, -53), sqrt_pi = 1.77245385090551602729;
    const long double sqrt_pi_l = 1.772453850905516027298167483341145183L;
    std::mt19937_64 g(3);
    for (double tol : {0.499, 0.2, 5e-3, 5e-4, 1e-5, 1e-8, 1e-19, 1e-60}) {
        for (double rc : {0.9, 1.3}) {
            const double alpha = (1.0 / rc) * std::sqrt(-std::log(2.0 * tol)), alpha2 = alpha * alpha;
            const double alpha3 = (double)((long double)alpha * alpha * alpha);
            std::vector<double> rows;
            const int n = ewald_rows(rc * rc * alpha2, rows);
            ok = ok && rows.size() == (size_t)2 * n * kEwaldRow;
            double worst[2] = {}, ratio[2] = {};
            auto pair = [&](double r, double sum[4]) {
                const double r2 = r * r;
                if (!(r2 < rc * rc)) return;
                const double rinv = 1.0 / std::sqrt(r2), s = alpha2 * r2;
                const int row = ewald_row((float)r2 * (float)alpha2);
                if (row >= n) {
                    ok = false;
                    return;
                }
                const double *c = rows.data() + (size_t)kEwaldRow * row;
                const double f = ewald_term(row, ewald_poly(c, r2, alpha2), alpha3, rinv * (rinv * rinv));
                const double e = ewald_term(row, ewald_poly(c + (size_t)kEwaldRow * n, r2, alpha2), alpha, rinv);
                const long double R = sqrtl((long double)r2), X = alpha * R;
                const long double el = erfcl(X) / R, fl = (erfcl(X) + 2 * X * expl(-X * X) / sqrt_pi_l) / (R * R * R);
                const double x = alpha * std::sqrt(r2);
                const double fd = rinv * rinv * rinv * (std::erfc(x) + 2 * x * std::exp(-x * x) / sqrt_pi);
                const double ed = rinv * std::erfc(x);
                const double d[4] = {(double)((f - fl) / fl), (double)((e - el) / el), (double)((fd - fl) / fl),
                                     (double)((ed - el) / el)};
                for (int k = 0; k < 4; ++k) sum[k] += d[k] * d[k];
                for (int k = 0; k < 2; ++k) worst[k] = std::max(worst[k], std::fabs(d[k]) / (ulp * (9 + 1.1 * s)));
            };
            for (int bin = 0; bin < 8; ++bin) {
                const double lo = std::max(0.02, rc * bin / 8), hi = rc * (bin + 1) / 8;
                std::uniform_real_distribution<double> u(lo, hi);
                double sum[4] = {};
                for (int k = 0; k < 4000; ++k) pair(u(g), sum);
                for (int k = 0; k < 2; ++k) ratio[k] = std::max(ratio[k], std::sqrt(sum[k] / sum[k + 2]));
            }
            double unused[4] = {};
            for (double s : {1.0 / 16, 1.0 / 8, 1.0, 2.0, 7.97, 8.0, 8.03, 40.0, alpha2 * rc * rc})
                for (double off : {-1e-7, -1e-15, 0.0, 1e-15, 1e-7}) pair(std::sqrt(s * (1 + off)) / alpha, unused);
            const bool good = worst[0] <= 1 && worst[1] <= 1 && ratio[0] <= 1.5 && ratio[1] <= 1.5;
            std::printf("tolerance %g cutoff %g: %d rows, worst of the bound: force %.2f energy %.2f, RMS over erfc's: %.2f %.2f%s\n",
                        tol, rc, n, worst[0], worst[1], ratio[0], ratio[1], good ? "" : " WRONG");
            ok = ok && good;
        }
    }
    std::printf("%s\n", ok ? "OK" : "FAILED");
    return ok ? 0 : 1;
}
