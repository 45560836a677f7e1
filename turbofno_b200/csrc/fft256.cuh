// 256-sample forward transform by eight adjacent lanes, truncated to 64 modes, with ONE exchange through shared
// memory: the alternative to forward_trunc32<8> where a kernel is bound by the load/store unit.
//
//   Lane r holds x[16 i + 2 r + q], i < 16, q < 2: sixteen-byte loads of adjacent samples (a group covers whole
//   128-byte lines).  With rho = 2 r + q = 4 a + b and k = k1 + 16 k2 (k1 < 16, k2 < 4):
//       F_rho[k1] = FFT16 over i                                                      in the lane
//       X[k] = sum_b W256^{b k} G_b[k],   G_b[k] = sum_a W4^{a k2} ( W64^{a k1} F_{4a+b}[k1] )
//            = (G_0 + W256^{2k} G_2) + W256^{k} (G_1 + W256^{2k} G_3)
//   Lane d collects all sixteen rho of k1 = 2 d, 2 d + 1 and ends with modes 2 d + e + 16 k2.
//
// Against forward_trunc32<8>: no table multiply (16 sixteen-byte reads that eight lanes do not share), no exchange
// rounds (112 shuffles and 32 complex multiply-adds), 16 instead of 32 global loads; 48 shared-memory accesses instead.
#pragma once
#include "fft32.cuh"

namespace tfno {

TFNO_HD constexpr int slot16(int k) { return 4 * (k & 3) + (k >> 2); }

template <int S, int K1>
TFNO_HD void twiddle_row16(float2* v) {          // v[4*K1 + n2] *= W16^{n2*K1}
    v[4 * K1 + 1] = twiddle32<S, 2, K1>(v[4 * K1 + 1]);
    v[4 * K1 + 2] = twiddle32<S, 4, K1>(v[4 * K1 + 2]);
    v[4 * K1 + 3] = twiddle32<S, 6, K1>(v[4 * K1 + 3]);
}
// 16-point transform, in registers.  In: v[n] = sample n.  Out: mode k in v[slot16(k)].
template <int S>
TFNO_HD void fft16(float2 (&v)[16]) {
#pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) dft4<S>(v[n2], v[4 + n2], v[8 + n2], v[12 + n2]);
    twiddle_row16<S, 1>(v); twiddle_row16<S, 2>(v); twiddle_row16<S, 3>(v);
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) dft4<S>(v[4 * k1], v[4 * k1 + 1], v[4 * k1 + 2], v[4 * k1 + 3]);
}

// Ten entries per k1: W64^{a k1} (a = 1..3), W256^{2 k1}, W256^{2 (k1 + 16)}, W256^{k1 + 16 k2} (k2 = 0..3), one unused.
// A pair of entries of the sixteen k1 is 256 contiguous bytes in the order [k1 % 2][k1 / 2]: eight lanes that want
// k1 = 2 d + e read 128 bytes.
constexpr int kTable256 = 16 * 10;
TFNO_HD constexpr int table256_index(int k1, int entry) { return (entry >> 1) * 32 + ((k1 & 1) * 8 + (k1 >> 1)) * 2 + (entry & 1); }
TFNO_HD void fill_table256(float2* tw, int tid, int nthreads) {
    for (int i = tid; i < kTable256; i += nthreads) {
        const int k1 = i / 10, j = i % 10;
        const int e = j < 3 ? 4 * (j + 1) * k1 : j < 5 ? 2 * (k1 + 16 * (j - 3)) : k1 + 16 * ((j - 5) & 3);
        tw[table256_index(k1, j)] = unit_root(e & 255, 256, -1.0f);
    }
}

// f[rho] = F_rho[k1].  out[k2] = X[k1 + 16 k2].  The factors of b are single table entries (constant W16^{b k2} times
// W256^{b k1}, added one after the other, put the result 7 % further from the exact transform: 1.03e-7 against 0.96e-7,
// forward_trunc32<8> 0.97e-7); those of k2 = 2, 3 in W256^{2k} are the ones of k2 = 0, 1 times -i.
TFNO_HD void combine256(float2 (&f)[16], const float2* __restrict__ table, int k1, float2 (&out)[4]) {
    const float2* tw = table + table256_index(k1, 0);
    const float4 t0 = *reinterpret_cast<const float4*>(tw), t1 = *reinterpret_cast<const float4*>(tw + 32);
    const float2 w1 = make_float2(t0.x, t0.y), w2 = make_float2(t0.z, t0.w), w3 = make_float2(t1.x, t1.y), v0 = make_float2(t1.z, t1.w);
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        f[4 + b] = cmul(f[4 + b], w1);
        f[8 + b] = cmul(f[8 + b], w2);
        f[12 + b] = cmul(f[12 + b], w3);
        dft4<-1>(f[b], f[4 + b], f[8 + b], f[12 + b]);                  // k2 at f[4*k2 + b]
    }
    const float4 t2 = *reinterpret_cast<const float4*>(tw + 64), t3 = *reinterpret_cast<const float4*>(tw + 96), t4 = *reinterpret_cast<const float4*>(tw + 128);
    const float2 v1 = make_float2(t2.x, t2.y);
    const float2 u[4] = {make_float2(t2.z, t2.w), make_float2(t3.x, t3.y), make_float2(t3.z, t3.w), make_float2(t4.x, t4.y)};
    const float2 v[4] = {v0, v1, make_float2(v0.y, -v0.x), make_float2(v1.y, -v1.x)};
#pragma unroll
    for (int k2 = 0; k2 < 4; ++k2)
        out[k2] = cmadd(cmadd(f[4 * k2], v[k2], f[4 * k2 + 2]), u[k2], cmadd(f[4 * k2 + 1], v[k2], f[4 * k2 + 3]));
}

#if defined(__CUDACC__)
// One quarter of the exchange: value(d) of every lane r goes to lane d, which receives those of r = 0..7 as
// got[2 r + q].  scratch: 64 elements of the group, [d][r] with the 16-byte pieces of a row permuted by d and
// the two rows of a pair swapped in odd groups, so that reads and writes cover all banks.
template <typename Value>
TFNO_D void exchange256(float2* scratch, int r, int odd_group, int q, float2 (&got)[16], Value value) {
#pragma unroll
    for (int d = 0; d < 8; ++d) scratch[(d ^ odd_group) * 8 + (((r >> 1) ^ (d >> 1)) << 1) + (r & 1)] = value(d);
    __syncwarp();
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const float4 p = *reinterpret_cast<const float4*>(scratch + (r ^ odd_group) * 8 + ((c ^ (r >> 1)) << 1));
        got[4 * c + q] = make_float2(p.x, p.y);
        got[4 * c + 2 + q] = make_float2(p.z, p.w);
    }
    __syncwarp();
}
#endif

}  // namespace tfno
