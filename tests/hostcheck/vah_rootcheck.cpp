// tests/hostcheck/vah_rootcheck.cpp -- host build of the closed root, the
// limiter in its bit form and the flux launches' work division, for
// tests/test_flux_division.py. Not part of the library, and never loaded by it.
#include <cmath>
#include <random>

#include "vah_march.cuh"

extern "C" {

// n random states and guesses: out[0] = states where the root is admitted and
// the guess accepted but the iteration falls back, out[1] = accepted, out[2] =
// iteration fallbacks, out[3] = largest relative difference of u_T over the
// accepted ones with u_T above 1e-10, out[4] = of e (relative to m0, the scale
// from which c0 = m0 - t^2 F m3 may cancel).
void rc_roots(long long n, unsigned seed, double *out) {
    std::mt19937_64 gen(seed);
    std::uniform_real_distribution<double> U(0, 1);
    std::normal_distribution<double> N;
    for (int k = 0; k < 5; ++k) out[k] = 0;
    for (long long it = 0; it < n; ++it) {
        const double t = 0.25 + 5 * U(gen), e = std::pow(10, -8 + 10 * U(gen));
        const double pl = e * (U(gen) < 0.8 ? U(gen) * 0.6 : U(gen) * 3 - 1), Pi = U(gen) < 0.5 ? 0.1 * e * N(gen) : 0.0;
        const double uT = U(gen) < 0.1 ? 0.0 : std::pow(10, -6 + 7.5 * U(gen)), ph = 6.283185307179586 * U(gen);
        const double ux = uT * std::cos(ph), uy = uT * std::sin(ph);
        const double un = U(gen) < 0.8 ? N(gen) * (U(gen) < 0.5 ? 0.3 : 2) / t : 0.0;
        const double ut = std::sqrt(1 + ux * ux + uy * uy + t * t * un * un);
        const double pt = 0.5 * (e - pl) + 1.5 * Pi, DP = pl - pt, F = 1 + ux * ux + uy * uy;
        const double amp = U(gen) < 0.5 ? 0 : std::pow(10, -6 + 6 * U(gen));  // distance from a consistent state
        vah::InvIn q;
        q.m0 = ((e + pt) * ut * ut - pt + DP * t * t * un * un / F) * (1 + 0.3 * amp * N(gen));
        q.m1 = (e + pt) * ut * ux + amp * e * N(gen);
        q.m2 = (e + pt) * ut * uy + amp * e * N(gen);
        q.m3 = ((e + pt) * ut * un + DP * ut * un / F) * (1 + amp * N(gen));
        q.pl = pl;
        q.bulk = Pi;
        const double r = U(gen);
        double w0 = uT;  // a neighbour's velocity, or anything
        if (r < 0.4) w0 = uT * (1 + 0.05 * N(gen));
        else if (r < 0.6) w0 = uT * std::pow(10, 2 * N(gen));
        else if (r < 0.8) w0 = std::pow(10, -6 + 8 * U(gen));
        else if (r < 0.9) w0 = 0;
        w0 = std::fabs(w0);
        vah::InvRoot root;
        vah::invert_root(t, q, root);
        vah::InvSetup s;
        vah::invert_setup(t, q, s);
        double u;
        const int st = vah::newton_uT(s, w0, u);
        out[2] += st != 0;
        if (!vah::newton_reaches(root, vah::newton_guess(w0, 0.0))) continue;
        out[1] += 1;
        if (st != 0) {
            out[0] += 1;
            continue;
        }
        const double v = u / std::sqrt(1 + u * u), C = 1 / std::sqrt(1 - 2 * root.s2 * root.inv);
        const double u_root = 2 * root.x2 / s.x * root.inv * C * s.mbt;
        if (u > 1e-10) out[3] = std::fmax(out[3], std::fabs(u_root - u) / u);
        out[4] = std::fmax(out[4], std::fabs(s.c0 - v * s.x * s.mbt - (root.c0 - root.s2)) / std::fabs(q.m0));
    }
}

// The edge state q + limited4 / 4 against q + approx_derivative / 2, both widths: mismatches.
long long rc_limiter(const double *x, const double *y, const double *z, long long n) {
    long long bad = 0;
    for (long long i = 0; i < n; ++i) {
        const double a = y[i] + 0.25 * vah::limited4(y[i] - x[i], z[i] - y[i], z[i] - x[i]);
        const double b = y[i] + 0.5 * vah::approx_derivative(x[i], y[i], z[i]);
        const float xf = (float)x[i], yf = (float)y[i], zf = (float)z[i];
        const float c = yf + 0.25f * vah::limited4(yf - xf, zf - yf, zf - xf);
        const float d = yf + 0.5f * vah::approx_derivative(xf, yf, zf);
        bad += !(a == b) || !(c == d);
    }
    return bad;
}

// How often flux_x's strips (width 0) or a march's strips own each interior
// cell or column: writes the smallest and largest count.
void rc_x_cover(int f32, int nx, int ny, int nk, int *lo, int *hi) {
    const int W = f32 ? 32 : 16, strips = f32 ? vah::flux_x_strips<float>(nx, ny, nk) : vah::flux_x_strips<double>(nx, ny, nk);
    const int ncx = nx + 4, total = nk * ny * ncx;
    int *n = new int[total]();
    for (int s = 0; s < strips; ++s)
        for (int pos = 1; pos <= W - 2; ++pos) {
            const int f = (W - 2) * s + 1 + pos;
            if (f < total) ++n[f];
        }
    *lo = 1 << 30;
    *hi = 0;
    for (int f = 0; f < total; ++f) {
        const int i = f % ncx;
        if (i < 2 || i > nx + 1) continue;
        *lo = n[f] < *lo ? n[f] : *lo;
        *hi = n[f] > *hi ? n[f] : *hi;
    }
    delete[] n;
}

int rc_march_strips(int f32, int columns) { return f32 ? vah::march_strips<float>(columns) : vah::march_strips<double>(columns); }

}  // extern "C"
