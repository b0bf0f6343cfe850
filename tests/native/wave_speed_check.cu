// Checks the exact form's wave speed (rusanov, physics.cuh) against the
// reference's expressions (getrusanov.f90:60-100) one by one, bit for bit, for
// ordinary states and for densities and fields near the ends of the format, where
// an operation saved elsewhere could overflow or lose bits.  Host code only
// (test infrastructure); exits non-zero at the first difference.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>

#include "physics.cuh"

using namespace sddc;

static double expected(const double *l, const double *r, double n0, double n1)
{
    const double mag = std::sqrt(n0 * n0 + n1 * n1), ux = n0 / mag, uy = n1 / mag;
    double p[2], vn[2];
    for (int s = 0; s < 2; s++) {
        const double *q = s ? r : l, i = 1.0 / q[0], u = i * q[1], v = i * q[2], w = i * q[3];
        const double b2 = (q[5] * q[5] + q[6] * q[6]) + q[7] * q[7];
        p[s] = (kGam - 1.0) * (((q[4] - 0.5 * q[0] * ((u * u + v * v) + w * w)) - b2 * 0.5) - 0.5 * (q[8] * q[8]));
        p[s] = p[s] + 0.5 * b2;
        p[s] = p[s] - 0.5 * b2;
        vn[s] = u * ux + v * uy;
    }
    const double Bx = 0.5 * (l[5] + r[5]), By = 0.5 * (l[6] + r[6]), Bz = 0.5 * (l[7] + r[7]), bn = Bx * ux + By * uy;
    const double ca = kGam * (p[0] + p[1]) / (l[0] + r[0]);
    const double cd = ((Bx * Bx + By * By) + Bz * Bz) / (0.5 * (l[0] + r[0])), cn = bn * bn / (0.5 * (l[0] + r[0]));
    const double cad = ca + cd, t = std::sqrt(cad * cad - 4.0 * ca * cn);
    return 0.5 * std::fabs(vn[0] + vn[1]) + std::sqrt(0.5 * ((ca + cd) + t));
}

int main()
{
    std::mt19937_64 rng(11);
    std::uniform_real_distribution<double> un(0.5, 1.0);
    // densities and fields as powers of two: ordinary, and pairs whose quotient is
    // ordinary though a doubled field energy or a halved density leaves the format
    const int ends[][2] = {{0, 0}, {-3, 2}, {530, 511}, {531, 512}, {520, 511}, {-1020, -500}, {-1022, -510}, {-1024, -511}, {-1074, -520}};
    for (auto &e : ends)
        for (int i = 0; i < 20000; i++) {
            double q[2][9];
            for (auto &s : q) {
                s[0] = std::ldexp(un(rng), e[0]);
                for (int k = 1; k < 4; k++) s[k] = 0.0;
                s[4] = 0.0;
                for (int k = 5; k < 8; k++) s[k] = std::ldexp(un(rng) - (i & 1 ? 0.75 : 0.0), e[1] - (k != 5 ? i % 7 : 0));
                s[8] = 0.0;
                if (e[0] == 0) s[1] = un(rng), s[2] = -un(rng), s[4] = 20.0 + un(rng);
            }
            const double n0 = un(rng), n1 = un(rng);
            double F[9], eig, um = 0.0;
            rusanov<double, true>(q[0], q[1], F, (double *)nullptr, n0, n1, 1, 1, 0.0, eig, um);
            const double want = expected(q[0], q[1], n0, n1);
            if (std::memcmp(&eig, &want, 8) && !(eig != eig && want != want)) {
                std::printf("2^%d, 2^%d: %a, not %a\n", e[0], e[1], eig, want);
                return 1;
            }
        }
    return 0;
}
