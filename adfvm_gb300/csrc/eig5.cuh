// Largest eigenvalue of a symmetric 5x5 matrix in FP64.
//
// Householder reduction to a tridiagonal matrix (Golub & Van Loan, Matrix Computations, the
// symmetric QR chapter), then Laguerre's method on its characteristic polynomial from above the
// spectrum, where it descends monotonically to the largest root of a polynomial with only real
// ones. The polynomial and its derivatives come from the three-term recurrence of the leading
// minors; above the spectrum each ratio of successive minors has one sign, so the recurrence is as
// accurate as the matrix entries. The start is the same iteration in FP32, which costs no FP64,
// raised by its error bound: two or three FP64 steps are left where the largest eigenvalue stands
// alone (convergence is cubic; laguerre5's estimate of what is left ends them), and a step leaves at
// most 3/8 of the distance where several coincide, so that its size ends those. About 250 FP64
// instructions on the GPU, whose FP64 pipe is the bound; cyclic Jacobi rotations to convergence took
// about 6,000 (k_visc_cell of 262,144 cells 2.13 -> 0.31 ms, with its face sums' shorter form).
#pragma once
#include <string.h>
#include "physics.cuh"

namespace afvm {

// Laguerre's step towards the largest root of the characteristic polynomial of the tridiagonal
// matrix with diagonal d and squared off-diagonals e2, from x above it (where the polynomial of
// degree five and its derivatives alternate in sign). last: whether what the step leaves is below
// the rounding of entries of size one. With d1 <= d2 <= ... the distances of x from the roots and
// s = sum d1/di, t = sum (d1/di)^2 over the other four, a step of a small s leaves
// d1 (t - s^2/4)/2 <= d1 s^2/2, and h = 2 p (p''/2) / (p'^2 - 2 p (p''/2)) = (2 s + s^2 - t)/(1 + t)
// is at least s as t <= s: what is left is at most step h^2/2. (h is large near several roots,
// so a step that lands among them is not taken for the last.)
template <typename F>
AFVM_HD F laguerre5(const F* d, const F* e2, F x, bool* last = nullptr) {
    F a = F(1), b = d[0] - x;              // minors of order i - 1 and i,
    F da = F(0), db = F(-1);               // their derivatives,
    F ha = F(0), hb = F(0);                // and half their second derivatives
    for (int i = 1; i < 5; i++) {
        const F t = d[i] - x, e = e2[i - 1];
        const F c = t * b - e * a;
        const F dc = (t * db - b) - e * da;
        const F hc = (t * hb - db) - e * ha;
        a = b; b = c;
        da = db; db = dc;
        ha = hb; hb = hc;
    }
    if constexpr (sizeof(F) == 4) {
        // (near five roots at once the squares below are not floats: 1e-35 where x is 2e-5 away)
        const F s = rcp(fabs(hb));
        b = b * s; db = db * s; hb = hb * s;
    }
    // n p / (p' - sqrt((n-1)^2 p'^2 - n (n-1) p p'')), n = 5. Five equal roots make the radicand zero: its
    // rounding error, some 20 units, would send x below them, so more than that is added (a step too
    // short by at most 5e-7 of itself in FP64, 0.011 in FP32, and by 2^-47 of itself at a simple root)
    constexpr F up = sizeof(F) == 4 ? F(16 + 0x1p-13) : F(16 + 0x1p-42);
    const F m = b * hb, g = db * db;
    const F r = up * g - F(40) * m;
    const F q = r > F(0) ? r * rsqrt_(r) : F(0);
    const F step = (F(5) * b) * rcp(db - q);
    if (last) {
        // step h^2 / 2 <= 1e-17, h = 2 m / (g - 2 m)
        const F k = g - F(2) * m;
        *last = step * (m * m) <= F(5e-18) * (k * k);
    }
    return step;
}

// conversions by integer instructions (on the device an FP64 conversion takes the FP64 pipe's time): x
// truncated to a float (zero below 2^-120; |x| < 2^100), and a float as a double (zero below 2^-126)
AFVM_HD float low(double x) {
    uint64_t b;
    memcpy(&b, &x, 8);
    const unsigned h = (unsigned)(b >> 32), l = (unsigned)b;
    const int e = (int)((h >> 20) & 0x7ffu) - 1023 + 127;
    const unsigned m = ((unsigned)e << 23) | ((h & 0xfffffu) << 3) | (l >> 29);
    const unsigned f = e < 7 ? 0u : (m | (h & 0x80000000u));
    float y;
    memcpy(&y, &f, 4);
    return y;
}
AFVM_HD double high(float x) {
    unsigned b;
    memcpy(&b, &x, 4);
    const unsigned e = (b >> 23) & 0xffu;
    const unsigned h = (b & 0x80000000u) | ((e + 896u) << 20) | ((b & 0x7fffffu) >> 3);
    const uint64_t f = e == 0u ? 0u : ((uint64_t)h << 32) | (b << 29);
    double y;
    memcpy(&y, &f, 8);
    return y;
}

// the upper triangle of a is used; NaN if an entry is not finite
AFVM_HD double max_eig5(const double a[5][5]) {
    // the largest magnitude, by the bits
    int64_t most = 0;
    for (int i = 0; i < 5; i++)
        for (int j = i; j < 5; j++) {
            int64_t b;
            memcpy(&b, &a[i][j], 8);
            b &= 0x7fffffffffffffffLL;
            most = b > most ? b : most;
        }
    const int e = (int)(most >> 52);
    if (most == 0) return 0.0;
    // the matrix scaled by a power of two to entries in [-2, 2]: the minors stay within 1e5, and in
    // FP32 those of x 4e-6 from five roots above 1e-27
    double scale, back;
    int64_t bits = (int64_t)(2046 - e) << 52;
    memcpy(&scale, &bits, 8);
    bits = e >= 2046 ? 0x7ff8000000000000LL : (int64_t)e << 52;
    memcpy(&back, &bits, 8);
    if (e >= 2046) return back;
    double s[5][5];
    for (int i = 0; i < 5; i++)
        for (int j = i; j < 5; j++) s[i][j] = a[i][j] * scale;
    double d[5], e2[4];
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (int k = 0; k < 3; k++) {
        // reflect column k below the diagonal onto its first entry
        const int m = 4 - k;               // its length
        double x0 = s[k][k + 1], tail = 0.0;
        for (int i = 1; i < m; i++) tail += s[k][k + 1 + i] * s[k][k + 1 + i];
        d[k] = s[k][k];
        const double n2 = x0 * x0 + tail;
        e2[k] = n2;
        // (a tail below 1e-40 of the matrix is no column to reflect)
        if (!(tail > 1e-80)) continue;
        const double norm = n2 * rsqrt_(n2);
        double v[4];
        v[0] = x0 + (x0 >= 0.0 ? norm : -norm);
        for (int i = 1; i < m; i++) v[i] = s[k][k + 1 + i];
        const double beta = rcp(norm * fabs(v[0]));          // 2 / v.v
        double p[4], pv = 0.0;
        for (int i = 0; i < m; i++) {
            double t = 0.0;
            for (int j = 0; j < m; j++) t += (j >= i ? s[k + 1 + i][k + 1 + j] : s[k + 1 + j][k + 1 + i]) * v[j];
            p[i] = beta * t;
            pv += p[i] * v[i];
        }
        const double h = 0.5 * beta * pv;
        for (int i = 0; i < m; i++) p[i] -= h * v[i];
        for (int i = 0; i < m; i++)
            for (int j = i; j < m; j++) s[k + 1 + i][k + 1 + j] -= v[i] * p[j] + p[i] * v[j];
    }
    d[3] = s[3][3];
    d[4] = s[4][4];
    e2[3] = s[3][4] * s[3][4];
    // FP32: from Gershgorin's bound
    float df[5], ef[4], x = -8.0f;
    for (int i = 0; i < 5; i++) df[i] = low(d[i]);
    for (int i = 0; i < 4; i++) ef[i] = low(e2[i]);
    for (int i = 0; i < 5; i++) {
        float r = df[i];
        if (i > 0) r += sqrtf(ef[i - 1]);
        if (i < 4) r += sqrtf(ef[i]);
        x = fmaxf(x, r);
    }
    x += 2e-5f;
    for (int it = 0; it < 40; it++) {
        const float step = laguerre5(df, ef, x);
        if (!(step > 4e-6f)) break;
        x -= step;
    }
    // FP64: from above it by more than its error
    double y = high(x) + 8e-5;
    for (int it = 0; it < 60; it++) {
        bool last;
        const double step = laguerre5(d, e2, y, &last);
        if (!(step > 2e-16)) break;
        y -= step;
        if (last) break;
    }
    return y * back;
}

}  // namespace afvm
