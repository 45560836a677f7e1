// Host-side check of the 256-sample forward transform of turbofno_b200/csrc/fft256.cuh (the exchange replayed over
// emulated lanes) against a direct double-precision DFT, next to the 32-point form of the same transform (fft32.cuh).
// Prints the largest absolute error and the relative rms errors of both.
#include <complex>
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "../../turbofno_b200/csrc/fft256.cuh"

using cd = std::complex<double>;
using namespace tfno;

static double urand() { return 2.0 * rand() / RAND_MAX - 1.0; }

static void one_exchange(const float2 (&x)[256], const float2* table, float2 (&X)[64]) {
    static float2 F[16][16];                                     // [rho][slot]
    for (int rho = 0; rho < 16; ++rho) {
        for (int i = 0; i < 16; ++i) F[rho][i] = x[16 * i + rho];
        fft16<-1>(F[rho]);
    }
    for (int k1 = 0; k1 < 16; ++k1) {
        float2 f[16], out[4];
        for (int rho = 0; rho < 16; ++rho) f[rho] = F[rho][slot16(k1)];
        combine256(f, table, k1, out);
        for (int k2 = 0; k2 < 4; ++k2) X[k1 + 16 * k2] = out[k2];
    }
}

static void lanes32(const float2 (&x)[256], const float2* table, float2 (&X)[64]) {
    constexpr int R = 8;
    static float2 v[R][32], t[R][32];
    for (int r = 0; r < R; ++r) {
        for (int n = 0; n < 32; ++n) v[r][n] = x[R * n + r];
        forward_local32<R>(v[r], table, r);
    }
    for (int r = 0; r < R; ++r)
        for (int j = 0; j < 32; ++j) t[r][j] = cmadd(v[r][j], round1_coef32<R>(r), v[r ^ 4][j]);
    for (int r = 0; r < R; ++r)
        for (int j = 0; j < 16; ++j) v[r][slot32(j)] = cadd(t[r][slot32(j)], t[r ^ 2][slot32(16 + j)]);
    for (int r = 0; r < R; ++r)
        for (int j = 0; j < 8; ++j) {
            const int keep = (r & 1) ? 8 + j : j;
            X[8 * r + j] = cadd(v[r][slot32(keep)], v[r ^ 1][slot32(keep)]);
        }
}

int main() {
    srand(11);
    std::vector<cd> root(256);
    for (int i = 0; i < 256; ++i) root[i] = std::polar(1.0, -2.0 * kPi * i / 256);
    alignas(16) static float2 t256[kTable256], t32[8 * 32];
    fill_table256(t256, 0, 1);
    fill_forward_table32<8>(t32, 0, 1);
    double err = 0, sq256 = 0, sq32 = 0, ref2 = 0;
    for (int trial = 0; trial < 400; ++trial) {
        float2 x[256], a[64], b[64];
        for (auto& e : x) e = make_float2((float)urand(), (float)urand());
        one_exchange(x, t256, a);
        lanes32(x, t32, b);
        for (int k = 0; k < 64; ++k) {
            cd ref = 0;
            for (int n = 0; n < 256; ++n) ref += cd(x[n].x, x[n].y) * root[(n * k) & 255];
            const double d = std::abs(cd(a[k].x, a[k].y) - ref);
            err = std::max(err, d);
            sq256 += d * d;
            sq32 += std::norm(cd(b[k].x, b[k].y) - ref);
            ref2 += std::norm(ref);
        }
    }
    printf("max %.3e\nrms256 %.4e\nrms32 %.4e\n", err, std::sqrt(sq256 / ref2), std::sqrt(sq32 / ref2));
    return 0;
}
