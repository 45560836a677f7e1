// Host-side check of turbofno_b200/csrc/fft_real.cuh (the exchange replayed over emulated lanes) against direct
// double-precision transforms: prints the relative rms errors of the forward and the inverse transform of 128 and 256 samples.
#include <complex>
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "../../turbofno_b200/csrc/fft_real.cuh"

using cd = std::complex<double>;
using namespace tfno;

static double urand() { return 2.0 * rand() / RAND_MAX - 1.0; }

template <int N> static void check() {
    constexpr int L = RealRows<N>::L, K1 = RealRows<N>::K1, Q = RealRows<N>::Q, M = RealRows<N>::M;
    alignas(16) static float2 tw[N / 2];
    fill_real_table<N>(tw, 0, 1);
    auto part_k1 = [](int part, int d) { return real_mode<N>(part, d); };
    double fe = 0, fr = 0, ie = 0, ir = 0;
    for (int trial = 0; trial < 200; ++trial) {
        // forward
        float a[2][N];
        for (auto& row : a) for (auto& e : row) e = (float)urand();
        static float2 v[L][Q][K1], f[L][2][16];
        for (int r = 0; r < L; ++r)
            for (int q = 0; q < Q; ++q) {
                for (int j = 0; j < K1; ++j) v[r][q][j] = make_float2(a[0][16 * j + Q * r + q], a[1][16 * j + Q * r + q]);
                real_inner<N, -1>(v[r][q]);
            }
        for (int d = 0; d < L; ++d) {
            for (int part = 0; part < 2; ++part)
                for (int r = 0; r < L; ++r)
                    for (int q = 0; q < Q; ++q) f[d][part][Q * r + q] = v[r][q][real_slot<N>(part_k1(part, d))];
            real_combine<N>(f[d][0], f[d][1], tw, d);
        }
        for (int d = 0; d < L; ++d)
            for (int part = 0; part < 2; ++part)
                for (int k2 = 0; k2 < M; ++k2) {
                    float2 got[2];
                    real_separate<N>(f[d][0], f[d][1], part, d == 0, k2, got[0], got[1]);
                    const int k = part_k1(part, d) + K1 * k2;
                    for (int row = 0; row < 2; ++row) {
                        cd ref = 0;
                        for (int n = 0; n < N; ++n) ref += 2.0 * a[row][n] * std::polar(1.0, -2.0 * kPi * ((n * k) % N) / N);
                        fe += std::norm(cd(got[row].x, got[row].y) - ref); fr += std::norm(ref);
                    }
                }
        // inverse
        float2 s[2][64];
        for (auto& row : s) for (auto& e : row) e = make_float2((float)urand(), (float)urand());
        for (int d = 0; d < L; ++d) {
            float2 m[2][2][M];                                   // [part][row]
            for (int part = 0; part < 2; ++part)
                for (int row = 0; row < 2; ++row)
                    for (int k2 = 0; k2 < M; ++k2) m[part][row][k2] = s[row][part_k1(part, d) + K1 * k2];
            for (auto& e : f[d][0]) e = make_float2(NAN, NAN);   // inputs that must not be read
            for (auto& e : f[d][1]) e = make_float2(NAN, NAN);
            real_join<N>(f[d][0], f[d][1], m[0][0], m[0][1], m[1][0], m[1][1], d == 0);
            real_spread<N>(f[d][0], f[d][1], tw, d);
        }
        for (int r = 0; r < L; ++r)
            for (int q = 0; q < Q; ++q) {
                for (int d = 0; d < L; ++d)
                    for (int part = 0; part < 2; ++part) v[r][q][part_k1(part, d)] = f[d][part][slot16(Q * r + q)];
                real_inner<N, 1>(v[r][q]);
                for (int j = 0; j < K1; ++j)
                    for (int row = 0; row < 2; ++row) {
                        const int n = 16 * j + Q * r + q;
                        double ref = s[row][0].x;
                        for (int k = 1; k < 64; ++k) ref += 2.0 * (cd(s[row][k].x, s[row][k].y) * std::polar(1.0, 2.0 * kPi * ((n * k) % N) / N)).real();
                        const float2 o = v[r][q][real_slot<N>(j)];
                        ie += std::pow((row ? o.y : o.x) - ref, 2); ir += ref * ref;
                    }
            }
    }
    printf("forward%d %.4e\ninverse%d %.4e\n", N, std::sqrt(fe / fr), N, std::sqrt(ie / ir));
}

int main() {
    srand(5);
    check<128>();
    check<256>();
    return 0;
}
