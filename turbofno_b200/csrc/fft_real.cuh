// Two real rows of N = 128 or 256 samples as one complex transform z = a + i b by L = N/32 adjacent lanes with ONE exchange
// through shared memory, forward (64 modes of each row) and inverse (from 64 modes of each).
//
//   n = rho + 16 j (rho < 16, j < K1 = N/16),  k = k1 + K1 k2 (k1 < K1, k2 < 16):
//       Z[k] = sum_rho W16^{rho k2} ( W_N^{rho k1} F_rho[k1] ),   F_rho = DFT over j
//   The rows are separated by Z[k] and Z[N-k].  Lane d takes k1 = d (part A) and k1 = K1 - d (part B; lane 0: K1/2), so that
//   both are in the same lane: N - k is the other part's 15 - k2 (lane 0: its own 16 - k2, or 15 - k2 of part B).  Part B is
//   kept under the number s = k2 + 1, which turns its factors into W_N^{rho (k1 - K1)}: the conjugates of part A's.
//   A lane holds Q = 16/L residues rho = Q r + q on the sample side: 8 (N = 256) or 16 (N = 128) contiguous bytes of a row.
//
// Against separating the rows before the exchange: half the exchanged values, and one combination of sixteen residues
// per k1 instead of one for each row.  The inverse, which took the 64 modes into every lane, reads each mode once.  1024
// images (1280 of 128 x 128), us, before and now: 256 x 256 forward 104 -> 85, inverse 115 -> 81 (46 at copy speed); 128 x 256 61 -> 49
// and 60 -> 40; 256 x 128 87 -> 64 and 77 -> 53; 128 x 128 57 -> 41 and 50 -> 34 (19).  Bound by issue slots and the load/store unit.
#pragma once
#include "fft256.cuh"

namespace tfno {

template <int N> struct RealRows {
    static_assert(N == 128 || N == 256, "two exchanged parts of sixteen values per lane");
    static constexpr int L = N / 32, K1 = N / 16, Q = 16 / L, M = 64 / K1;      // M: kept k2 of a part
    static constexpr int SCRATCH = 8 * L;                                        // exchanged values per group of lanes
};
// register of mode k of the K1-point transform in the lane
template <int N> TFNO_HD constexpr int real_slot(int k) { return N == 256 ? slot16(k) : k; }
template <int N, int S> TFNO_HD void real_inner(float2 (&v)[N / 16]) {
    if constexpr (N == 256) fft16<S>(v);
    else fft8<S>(v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], make_odd_sign(1.0f));
}

// Factors W_N^{rho d} of lane d; those of rho, rho + 1 of the L lanes are adjacent.  N/2 entries.  Part B's are their conjugates;
// lane 0, whose part A needs none, has those of its part B: W_N^{rho K1/2}.
template <int N> TFNO_HD constexpr int real_table_index(int d, int rho) { return ((rho >> 1) * RealRows<N>::L + d) * 2 + (rho & 1); }
template <int N> TFNO_HD void fill_real_table(float2* tw, int tid, int nthreads) {
    constexpr int L = RealRows<N>::L, K1 = RealRows<N>::K1;
    for (int i = tid; i < N / 2; i += nthreads) {
        const int d = i / 16, rho = i % 16;
        tw[real_table_index<N>(d, rho)] = unit_root((rho * (d ? d : K1 / 2)) & (N - 1), N, -1.0f);
    }
    static_assert(16 * L == N / 2, "sixteen factors per lane");
}
// first k of a part
template <int N> TFNO_HD int real_mode(int part, int d) { return part == 0 ? d : d ? RealRows<N>::K1 - d : RealRows<N>::K1 / 2; }

TFNO_HD float2 cmul_conj(float2 a, float2 b) { return make_float2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y); }
// the parts' f[at(rho)] times their factors (forward) or the conjugates of them (inverse)
template <int N, bool INVERSE, typename At>
TFNO_HD void real_twiddle(float2 (&fa)[16], float2 (&fb)[16], const float2* tw, int d, At at) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float4 t = *reinterpret_cast<const float4*>(tw + real_table_index<N>(d, 2 * j));
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (j == 0 && h == 0) continue;
            const float2 w = h ? make_float2(t.z, t.w) : make_float2(t.x, t.y);
            const float2 wa = d ? w : make_float2(1.f, 0.f);
            float2 &a = fa[at(2 * j + h)], &b = fb[at(2 * j + h)];
            a = INVERSE ? cmul_conj(a, wa) : cmul(a, wa);
            b = INVERSE ? cmul(b, w) : cmul_conj(b, w);
        }
    }
}

// ---- forward, after the exchange: f[rho] of the parts -> k2 (part A) and s (part B) at f[slot16(.)] ----
template <int N> TFNO_HD void real_combine(float2 (&fa)[16], float2 (&fb)[16], const float2* tw, int d) {
    real_twiddle<N, false>(fa, fb, tw, d, [](int rho) { return rho; });
    fft16<-1>(fa);
    fft16<-1>(fb);
}
// mode real_mode(part, d) + K1 k2 of rows a and b, both times 2
template <int N>
TFNO_HD void real_separate(const float2 (&fa)[16], const float2 (&fb)[16], int part, bool lane0, int k2, float2& a, float2& b) {
    const float2 own = part == 0 ? fa[slot16(k2)] : fb[slot16(k2 + 1)];
    const float2 mb = fb[slot16((16 - k2) & 15)];
    const float2 ma = part == 0 ? fa[slot16((16 - k2) & 15)] : fa[slot16(15 - k2)];
    const float2 mirror = (part == 0) == lane0 ? ma : mb;
    a = make_float2(own.x + mirror.x, own.y - mirror.y);
    b = make_float2(own.y + mirror.y, mirror.x - own.x);
}

// ---- inverse, before the exchange ----
// Modes a[k2], b[k2] of the two rows, k = real_mode(part, d) + K1 k2, into the inputs k2 / s of the parts (in order).
// Mode 0 enters once.  N = 256: the inputs of no mode are left out (real_expand skips them), N = 128: only k = 64.
template <int N>
TFNO_HD void real_join(float2 (&fa)[16], float2 (&fb)[16], const float2 (&aA)[RealRows<N>::M], const float2 (&bA)[RealRows<N>::M],
                       const float2 (&aB)[RealRows<N>::M], const float2 (&bB)[RealRows<N>::M], bool lane0) {
    constexpr int M = RealRows<N>::M;
    float2 mA[M], mB[M];                                     // conj(a) + i conj(b)
#pragma unroll
    for (int k2 = 0; k2 < M; ++k2) {
        fa[k2] = make_float2(aA[k2].x - bA[k2].y, aA[k2].y + bA[k2].x);
        fb[k2 + 1] = make_float2(aB[k2].x - bB[k2].y, aB[k2].y + bB[k2].x);
        mA[k2] = make_float2(aA[k2].x + bA[k2].y, bA[k2].x - aA[k2].y);
        mB[k2] = make_float2(aB[k2].x + bB[k2].y, bB[k2].x - aB[k2].y);
    }
    if (lane0) fa[0] = make_float2(aA[0].x, bA[0].x);
#pragma unroll
    for (int k2 = 0; k2 < M; ++k2) {
        fb[(16 - k2) & 15] = lane0 ? mB[k2] : mA[k2];
        fa[15 - k2] = !lane0 ? mB[k2] : k2 + 1 < M ? mA[(k2 + 1) % M] : make_float2(0.f, 0.f);
    }
}
// the sixteen-point transform of a part's inputs; of 256 samples, inputs 4..11 (part B: 5..12) are zero
template <int N, int PART>
TFNO_HD void real_expand(float2 (&f)[16]) {
    if constexpr (N == 128) fft16<1>(f);
    else {
#pragma unroll
        for (int n2 = 0; n2 < 4; ++n2) {
            const bool second = PART == 1 && n2 == 0;         // inputs 0 and 4; elsewhere n2 and 12 + n2
            const float2 b0 = f[n2], t = second ? f[4] : f[12 + n2];
            const float2 it = second ? make_float2(-t.y, t.x) : make_float2(t.y, -t.x);
            f[n2] = cadd(b0, t); f[8 + n2] = csub(b0, t); f[4 + n2] = cadd(b0, it); f[12 + n2] = csub(b0, it);
        }
        twiddle_row16<1, 1>(f); twiddle_row16<1, 2>(f); twiddle_row16<1, 3>(f);
#pragma unroll
        for (int k1 = 0; k1 < 4; ++k1) dft4<1>(f[4 * k1], f[4 * k1 + 1], f[4 * k1 + 2], f[4 * k1 + 3]);
    }
}
template <int N>
TFNO_HD void real_spread(float2 (&fa)[16], float2 (&fb)[16], const float2* tw, int d) {          // result for rho at f[slot16(rho)]
    real_expand<N, 0>(fa);
    real_expand<N, 1>(fb);
    real_twiddle<N, true>(fa, fb, tw, d, [](int rho) { return slot16(rho); });
}

#if defined(__CUDACC__)
// value(e) of every lane r goes to lane e of its group, which receives got(r, value).  256: exchange256's layout.  128: two
// values at a time, [e][r] 16-byte pieces permuted by e, rows swapped in odd groups: reads and writes cover all banks.
template <typename Value, typename Got>
TFNO_D void real_exchange256(float2* scratch, int r, int odd_group, Value value, Got got) {
#pragma unroll
    for (int e = 0; e < 8; ++e) scratch[(e ^ odd_group) * 8 + (((r >> 1) ^ (e >> 1)) << 1) + (r & 1)] = value(e);
    __syncwarp();
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const float4 p = *reinterpret_cast<const float4*>(scratch + (r ^ odd_group) * 8 + ((c ^ (r >> 1)) << 1));
        got(2 * c, make_float2(p.x, p.y));
        got(2 * c + 1, make_float2(p.z, p.w));
    }
    __syncwarp();
}
template <typename Value, typename Got>
TFNO_D void real_exchange128(float2* scratch, int r, int odd_group, Value value, Got got) {
    float4* s = reinterpret_cast<float4*>(scratch);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float2 a = value(e, 0), b = value(e, 1);
        s[(e ^ odd_group) * 4 + (r ^ e)] = make_float4(a.x, a.y, b.x, b.y);
    }
    __syncwarp();
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const float4 p = s[(r ^ odd_group) * 4 + (c ^ r)];
        got(c, 0, make_float2(p.x, p.y));
        got(c, 1, make_float2(p.z, p.w));
    }
    __syncwarp();
}

// Samples v[q][j] of rho = Q r + q (consumed) -> the combined parts
template <int N>
TFNO_D void real_forward(float2 (&v)[RealRows<N>::Q][N / 16], const float2* tw, float2* scratch, int r, int odd_group, float2 (&fa)[16], float2 (&fb)[16]) {
    constexpr int K1 = RealRows<N>::K1, Q = RealRows<N>::Q;
#pragma unroll
    for (int q = 0; q < Q; ++q) real_inner<N, -1>(v[q]);
#pragma unroll
    for (int part = 0; part < 2; ++part) {
        float2 (&f)[16] = part ? fb : fa;
#pragma unroll
        for (int q = 0; q < Q; q += (N == 256 ? 1 : 2)) {
            auto k1 = [&](int e) { return part == 0 ? e : e ? K1 - e : K1 / 2; };
            if constexpr (N == 256)
                real_exchange256(scratch, r, odd_group, [&](int e) { return v[q][real_slot<N>(k1(e))]; }, [&](int c, float2 x) { f[2 * c + q] = x; });
            else
                real_exchange128(scratch, r, odd_group, [&](int e, int h) { return v[q + h][real_slot<N>(k1(e))]; }, [&](int c, int h, float2 x) { f[4 * c + q + h] = x; });
        }
    }
    real_combine<N>(fa, fb, tw, r);
}
// Inputs of the parts (consumed) -> samples of rho = Q r + q: j at v[q][real_slot<N>(j)]
template <int N>
TFNO_D void real_inverse(float2 (&fa)[16], float2 (&fb)[16], const float2* tw, float2* scratch, int r, int odd_group, float2 (&v)[RealRows<N>::Q][N / 16]) {
    constexpr int K1 = RealRows<N>::K1, Q = RealRows<N>::Q;
    real_spread<N>(fa, fb, tw, r);
#pragma unroll
    for (int part = 0; part < 2; ++part) {
        const float2 (&f)[16] = part ? fb : fa;
#pragma unroll
        for (int q = 0; q < Q; q += (N == 256 ? 1 : 2)) {
            auto k1 = [&](int e) { return part == 0 ? e : e ? K1 - e : K1 / 2; };
            if constexpr (N == 256)
                real_exchange256(scratch, r, odd_group, [&](int e) { return f[slot16(2 * e + q)]; }, [&](int c, float2 x) { v[q][k1(c)] = x; });
            else
                real_exchange128(scratch, r, odd_group, [&](int e, int h) { return f[slot16(4 * e + q + h)]; }, [&](int c, int h, float2 x) { v[q + h][k1(c)] = x; });
        }
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) real_inner<N, 1>(v[q]);
}
#endif

}  // namespace tfno
