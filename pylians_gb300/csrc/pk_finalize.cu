// Spectra from the float64 sums of pyl_pk_bin, on the host: Pk_library.pyx:384-421 (Pk) and
// :740-796 (XPk).  One pass over the bins writes every result array, in the order of
// operations of those lines.  As numpy expressions (a temporary for each operation, a
// scatter for kpar and kper) four fields of 128^3 took 0.25 ms, two of 1023^3 7.0 ms for
// 0.08 and 1.2 ms here; Pk of 128^3 0.29 -> 0.20 ms, XPk of two 512^3 5.44 -> 4.05 ms.
// Bound by the pages of the results (372,000 k_par/k_per bins at 1024^3) and the divisions.
#include <cmath>

#include "common.cuh"

extern "C" int pyl_pk_finalize(const double *sums, const double *geom, int dims, int n_fields, int n_cross,
                               const double *consts, double *const *out)
{
    PYL_CHECK_ARG(sums && geom && consts && out, "null pointer");
    PYL_CHECK_ARG(dims >= 1 && n_fields >= 1 && n_cross >= -1, "bad sizes");
    const double kF = consts[0], kN2 = consts[1], fact = consts[2], pi = consts[3], four_pi2 = consts[4];
    const int F = n_fields, X = n_cross < 0 ? 0 : n_cross, C = F + F * (F - 1) / 2;
    const int FO = n_cross < 0 ? 1 : F;                     // Pk keeps its field only
    const int middle = dims / 2;
    const long long nb1 = middle + 1, nper = (long long)std::sqrt((double)middle * middle * 2.0) + 1;
    const long long nb3 = (long long)std::sqrt((double)middle * middle * 3.0) + 1, nb2 = nb1 * nper;
    const double *P3 = sums, *PH = P3 + nb3 * 3 * C, *P1 = PH + nb3 * F, *P2 = P1 + nb1 * C;
    const double *K1 = geom, *N1 = K1 + nb1, *N2 = N1 + nb1, *K3 = N2 + nb2, *N3 = K3 + nb3;

    for (long long i = 1; i < nb1; i++) {
        const double k = K1[i] / N1[i] * kF;
        const volatile double k2 = k * k;                   // rounded: no fused subtraction
        const double kper = std::sqrt(kN2 - k2);
        const double area = pi * (kper * kper) / N1[i] / four_pi2;
        out[0][i - 1] = k;
        out[1][i - 1] = N1[i];
        for (int c = 0; c < FO; c++) out[2][(i - 1) * FO + c] = P1[i * C + c] * fact * area;
        for (int c = 0; c < X; c++) out[3][(i - 1) * X + c] = P1[i * C + F + c] * fact * area;
    }
    for (long long q = 0; q < nper; q++) {
        const double kp = 0.5 * (double)(2 * q + 1) * kF;
        double *kpar = out[4] + q * nb1, *kper = out[5] + q * nb1;
        for (long long i = 0; i < nb1; i++) {
            kpar[i] = 0.5 * (double)(2 * i + 1) * kF;
            kper[i] = kp;
        }
    }
    for (long long b = 0; b < nb2; b++) {
        const double n = N2[b];
        out[6][b] = n;
        for (int c = 0; c < FO; c++) out[7][b * FO + c] = P2[b * C + c] * fact / n;
        for (int c = 0; c < X; c++) out[8][b * X + c] = P2[b * C + F + c] * fact / n;
    }
    for (long long i = 1; i < nb3; i++) {
        const double n = N3[i];
        out[9][i - 1] = K3[i] / n * kF;
        out[10][i - 1] = n;
        for (int l = 0; l < 3; l++) {                       // the l = 0 sums times 1: the same bits
            const double legendre = l == 0 ? 1.0 : l == 1 ? 5.0 : 9.0;
            const double *s = P3 + (i * 3 + l) * C;
            for (int c = 0; c < FO; c++) out[11][((i - 1) * 3 + l) * FO + c] = s[c] * legendre / n * fact;
            for (int c = 0; c < X; c++) out[12][((i - 1) * 3 + l) * X + c] = s[F + c] * legendre / n * fact;
        }
        if (n_cross < 0) out[13][i - 1] = PH[i * F] / n * fact;
    }
    return PYL_OK;
}
