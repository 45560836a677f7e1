// Channel contractions of compact spectra, one product per retained mode, and the gradients of the
// weights.  All of them are
//
//     O[i, j, m] = scale * sum_r  P[r, i, m] * conj?(Q[r, j, m])          (or the conjugate of it)
//
//   layer        C[n, b, m]  = alpha sum_k A[k, b, m] W[k, n, m]              i = b, j = n, r = k
//   grad of x    Gx[k, b, m] = alpha sum_n G[n, b, m] conj(W[k, n, m])        i = b, j = k, r = n
//   grad of W    dW[k, n, m] = s     sum_b conj(X[k, b, m]) G[n, b, m]        i = k, j = n, r = b
//   the same for weights shared by all modes: the sum also runs over m.  (b, m / 8) is then the index r
//                of a problem of eight modes, whose results are added at the end.
//
// The reference contracts with one K x N matrix shared by all modes
// (fusion_variants/1D_E_baseline/cgemm.cuh:42-43, B[k + n*K]); per-mode matrices are the extension its
// README names as the FNO use case.
//
// On the tensor cores through mma.sync m16n8k8 (tf32), every FP32 value split into two tf32 parts and three products
// kept (hi*hi + lo*hi + hi*lo), but for sums of few terms (PmProducts).  Fragments live in registers, so the operands are
// split on the way from the ring to the multiplier, each value once; tcgen05 would want both parts of every matrix written
// back to shared memory, one mode at a time, for products of 64 x 64 x (a few rows) each.  The tensor cores truncate when
// they accumulate, so a chain covers the eight terms of one step only and the steps are added in FP32: closer to the exact
// sums than chains of 24 FP32 FMAs and more (whole layer against 64-bit results: 1D training step 2.4e-7 -> 2.1e-7, real 2D
// field 2.9e-7 -> 2.6e-7).  Operands below 2^-115 lose the last bits of their low parts.
//
// What bounds it (2D, 4096 modes, K = N = 64; us, with the FP32 kernel before it): layer of 1 row 36 (36), 16 rows 51 (73), 20
// rows 66 (94), 64 rows 172 (242).  1D, 64 modes: 16 rows 7 (21), 512 rows 28 (37).  Not ahead everywhere: 40 -> 128 channels, 2
// rows 39.4 (37.4), 4 rows 41.6 (37.9).  Up to 8 rows the 134 MB of weights (20 us at copy speed); beyond that the multiplier,
// 55 % busy (20 rows: 33 us at 512 multiply-adds a cycle), with the latencies of a step (load, split, chain of six) behind
// four warps per scheduler.
// Tried: persistent CTAs whose ring runs on across tiles (79 us at 20 rows: 3.5 tiles per CTA are dealt worse than by the
// hardware), tiles of 16 columns with three CTAs per SM (71), all loads of a step ahead of its products (68).
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include "common.cuh"

namespace tfno {

constexpr int kPmCols = 32;            // columns j per CTA
constexpr int kPmThreads = 256;
constexpr int kPmTerms = 8;            // values of r per ring stage = depth of a matrix instruction
constexpr int kPmStages = 3;
// PM_SPLIT: two tf32 parts, three products; PM_FULL: four products; PM_FMA: FP32 multiply-adds (rule: permode.cu)
enum PmProducts { PM_SPLIT, PM_FULL, PM_FMA };
constexpr int kPmSumTile = 64;         // gradient of shared weights: rows i and columns j per CTA
constexpr int kPmSumTerms = 4;         // and r per ring stage (each eight modes deep)

template <int NT> __host__ __device__ constexpr int pm_stage_bytes() { return kPmTerms * (8 * NT + kPmCols) * kPmModes * 8; }
template <int NT> __host__ __device__ constexpr int pm_smem_bytes() { return kPmStages * pm_stage_bytes<NT>(); }
constexpr int kPmSumStageBytes = 2 * kPmSumTile * kPmSumTerms * kPmModes * 8;
constexpr int kPmSumSmemBytes = kPmStages * kPmSumStageBytes;

// copies `bytes` (16 or 8), or zeros when !live (the source is not read then)
__device__ __forceinline__ void pm_copy16(uint32_t dst, const void* src, bool live) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void pm_copy8(uint32_t dst, const void* src, bool live) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(live ? 8 : 0) : "memory");
}
__device__ __forceinline__ float4 pm_load16(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ float2 pm_load8(uint32_t addr) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr));
    return v;
}
// v = hi + lo, hi rounded to tf32 by an add and a mask and at most the largest finite tf32 (the last values below FLT_MAX would
// round to infinity, with a rest of minus infinity, and finite products would become NaN); infinities and NaNs are passed on in
// lo.  The bound costs up to 0.4 us of a small layer (64 signals of 128 samples 19.7 -> 20.1 us, training step of 512 of 512
// samples 246.0 -> 246.0).  The multiplier drops the low 13 bits of an operand: at most the last of lo's 12 bits.
__device__ __forceinline__ void pm_split(float v, uint32_t& hi, uint32_t& lo) {
    float h;
    asm("min.xorsign.abs.f32 %0, %1, %2;" : "=f"(h) : "f"(__uint_as_float((__float_as_uint(v) + 0x1000u) & 0xffffe000u)), "f"(__uint_as_float(0x7f7fe000u)));
    hi = __float_as_uint(h);
    lo = __float_as_uint(v - h);
}
__device__ __forceinline__ void pm_mma(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
__device__ __forceinline__ void pm_mma_first(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {      // d = a b
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(0.f));
}
// The two parts of a fragment of one matrix (real or imaginary).  Q is the 16-row operand: lane 4 g + t holds rows g, g + 8 at
// terms t, t + 4; P the 8-column one: column g at terms t, t + 4.
struct PmFragQ { uint32_t hi[4], lo[4]; };
struct PmFragP { uint32_t hi[2], lo[2]; };
__device__ __forceinline__ PmFragP pm_negated(const PmFragP& f) {
    PmFragP n;
#pragma unroll
    for (int i = 0; i < 2; ++i) { n.hi[i] = f.hi[i] ^ 0x80000000u; n.lo[i] = f.lo[i] ^ 0x80000000u; }
    return n;
}
// sum += P conj?(Q) over eight terms, the small products first.
// FULL: lo*lo too, and hi*hi of the two parts apart from the rest, so that what the tensor cores truncate is small or exact.
struct PmSum { float2 re[2], im[2]; };             // a fragment of results: lane 4 g + t holds columns 2 t, 2 t + 1 of rows g, g + 8
template <bool CONJ_Q, bool FULL>
__device__ __forceinline__ void pm_step(PmSum& sum, const PmFragQ& qr, const PmFragQ& qi, const PmFragP& pr, const PmFragP& pi, const PmFragP& n) {
    // Q: re = Pr Qr - Pi Qi, im = Pi Qr + Pr Qi, n = -Pi;  conj(Q): re = Pr Qr + Pi Qi, im = Pi Qr - Pr Qi, n = -Pr
    const PmFragP &re2 = CONJ_Q ? pi : n, &im2 = CONJ_Q ? n : pr;
    float a[4], b[4];
    if constexpr (FULL) {
        pm_mma_first(a, qr.lo, pr.lo); pm_mma_first(b, qr.lo, pi.lo);
        pm_mma(a, qi.lo, re2.lo); pm_mma(b, qi.lo, im2.lo);
        pm_mma(a, qr.lo, pr.hi);  pm_mma(b, qr.lo, pi.hi);
    } else {
        pm_mma_first(a, qr.lo, pr.hi); pm_mma_first(b, qr.lo, pi.hi);
    }
    pm_mma(a, qi.lo, re2.hi); pm_mma(b, qi.lo, im2.hi);
    pm_mma(a, qr.hi, pr.lo);  pm_mma(b, qr.hi, pi.lo);
    pm_mma(a, qi.hi, re2.lo); pm_mma(b, qi.hi, im2.lo);
    if constexpr (FULL) {
        float c[4], d[4], e[4], f[4];
        pm_mma_first(c, qr.hi, pr.hi);  pm_mma_first(d, qr.hi, pi.hi);
        pm_mma_first(e, qi.hi, re2.hi); pm_mma_first(f, qi.hi, im2.hi);
#pragma unroll
        for (int h = 0; h < 4; h += 2) {
            const float2 re = __fadd2_rn(__fadd2_rn(make_float2(c[h], c[h + 1]), make_float2(e[h], e[h + 1])), make_float2(a[h], a[h + 1]));
            const float2 im = __fadd2_rn(__fadd2_rn(make_float2(d[h], d[h + 1]), make_float2(f[h], f[h + 1])), make_float2(b[h], b[h + 1]));
            a[h] = re.x; a[h + 1] = re.y; b[h] = im.x; b[h + 1] = im.y;
        }
    } else {
        pm_mma(a, qr.hi, pr.hi);  pm_mma(b, qr.hi, pi.hi);
        pm_mma(a, qi.hi, re2.hi); pm_mma(b, qi.hi, im2.hi);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        sum.re[h] = __fadd2_rn(sum.re[h], make_float2(a[2 * h], a[2 * h + 1]));
        sum.im[h] = __fadd2_rn(sum.im[h], make_float2(b[2 * h], b[2 * h + 1]));
    }
}

// ---- one product per mode ----
// A CTA takes eight adjacent modes, 32 columns j and 8 NT rows i, a warp one mode of them.  Stages of eight r travel by
// 16-byte asynchronous copies through a ring of kPmStages; the 16-byte pieces of a line are permuted by r % 4, so that the
// sixteen lanes of a half-warp (four lines, four r) meet two by two.  The results leave through shared memory, as whole
// 64-byte lines.
// CONJ_Q: Q enters conjugated.  CONJ_O: the sum is conjugated before it is scaled (conj(P) Q = conj(P conj(Q))).
// MODE: how the products are made (see PmProducts).
template <int NT, bool CONJ_Q, bool CONJ_O, PmProducts MODE>
__global__ void __launch_bounds__(kPmThreads, NT == 1 ? 3 : 2) cgemm_permode_kernel(PerModeParams p) {
    constexpr int ROWS = 8 * NT, LINES = ROWS + kPmCols, STAGE = pm_stage_bytes<NT>(), MT = kPmCols / 16;
    static_assert(ROWS * kPmCols * 64 <= pm_smem_bytes<NT>(), "the results pass through the ring");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // CTAs that differ only in their rows i or columns j are neighbours: they share Q or P, which the L2 then serves
    const int iblocks = (p.I + ROWS - 1) / ROWS, jblocks = p.J / kPmCols;
    long long item = blockIdx.x;
    const int i0 = (int)(item % iblocks) * ROWS; item /= iblocks;
    const int j0 = (int)(item % jblocks) * kPmCols; item /= jblocks;
    const int split = (int)(item % p.splits); item /= p.splits;
    const long long m0 = item * kPmModes;
    const long long r0 = split * p.split_len;
    const long long r1 = (r0 + p.split_len < p.red) ? r0 + p.split_len : p.red;
    const int terms = r1 > r0 ? (int)(r1 - r0) : 0, steps = (terms + kPmTerms - 1) / kPmTerms;
    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(smem_raw);

    // copies: warp w brings the lines of term w of a stage, eight lines (512 bytes) at a time.  A copy of no bytes (rows
    // past I, terms past the end) fills with zeros and does not look at its source.
    const int c_line = lane >> 2, c_piece = lane & 3;
    const uint32_t c_dst = ring + (uint32_t)((warp * LINES + c_line) * 64 + ((c_piece ^ (warp & 3)) << 4));
    const float2* p_src = p.p + (r0 + warp) * p.p_sr + (long long)(i0 + c_line) * p.p_si + m0 + 2 * c_piece;
    const float2* q_src = p.q + (r0 + warp) * p.q_sr + (long long)(j0 + c_line) * p.q_sj + m0 + 2 * c_piece;
    auto fetch = [&](int step) {
        if (step < steps) {
            const uint32_t stage = (uint32_t)(step % kPmStages) * STAGE, dst = c_dst + stage;
            const bool live = step * kPmTerms + warp < terms;
#pragma unroll
            for (int l = 0; l < NT; ++l) pm_copy16(dst + l * 512, p_src + 8 * l * p.p_si, live && i0 + 8 * l + c_line < p.I);
            if (p.q_vec) {
#pragma unroll
                for (int l = 0; l < kPmCols / 8; ++l) pm_copy16(dst + (ROWS + 8 * l) * 64, q_src + 8 * l * p.q_sj, live);
            } else {
                // modes that are not adjacent, or lines on odd addresses: eight bytes at a time
                const float2* term = p.q + (r0 + (long long)step * kPmTerms + warp) * p.q_sr;
#pragma unroll 1
                for (int i = lane; i < kPmCols * 8; i += 32) {
                    const int mode = i & 7, line = i >> 3;
                    const uint32_t at = (uint32_t)((warp * LINES + ROWS + line) * 64 + (((mode >> 1) ^ (warp & 3)) << 4) + (mode & 1) * 8);
                    pm_copy8(ring + stage + at, term + (long long)(j0 + line) * p.q_sj + (m0 + mode) * p.q_sm, live);
                }
            }
            p_src += kPmTerms * p.p_sr;
            q_src += kPmTerms * p.q_sr;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    const int g = lane >> 2, t = lane & 3;
    const uint32_t frag = ring + (uint32_t)((t * LINES + g) * 64 + (((warp >> 1) ^ t) << 4) + (warp & 1) * 8);
    constexpr uint32_t HALF = 4 * LINES * 64;                    // terms t + 4
    PmSum acc[MODE == PM_FMA ? 1 : NT][MT];
    // PM_FMA: a lane has one mode, rows row + 4 a (adjacent lines of a half-warp cover all banks) and four columns
    const int mode = lane & 7, row = lane >> 3, col = 4 * warp;
    float2 sum[MODE == PM_FMA ? 2 * NT : 1][4];
    if constexpr (MODE == PM_FMA) {
#pragma unroll
        for (int i = 0; i < 8 * NT; ++i) (&sum[0][0])[i] = make_float2(0.f, 0.f);
    } else {
#pragma unroll
        for (int i = 0; i < NT * MT; ++i) (&acc[0][0])[i] = PmSum{};
    }
    follow_previous_kernel();
    admit_next_kernel();
#pragma unroll
    for (int s = 0; s < kPmStages - 1; ++s) fetch(s);
#pragma unroll 1
    for (int step = 0; step < steps; ++step) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kPmStages - 2) : "memory");
        __syncthreads();                          // this stage has arrived; everybody has left the one refilled next
        fetch(step + kPmStages - 1);
        if constexpr (MODE == PM_FMA) {
            const int last = terms - step * kPmTerms < kPmTerms ? terms - step * kPmTerms : kPmTerms;
            const uint32_t st = ring + (uint32_t)(step % kPmStages) * STAGE + (uint32_t)(mode & 1) * 8;
#pragma unroll 1
            for (int r = 0; r < last; ++r) {
                const uint32_t at = st + (uint32_t)(r * LINES * 64 + (((mode >> 1) ^ (r & 3)) << 4));
                float2 q[4];
#pragma unroll
                for (int b = 0; b < 4; ++b) q[b] = pm_load8(at + (uint32_t)(ROWS + col + b) * 64);
#pragma unroll
                for (int a = 0; a < 2 * NT; ++a) {
                    const float2 v = pm_load8(at + (uint32_t)(row + 4 * a) * 64);
#pragma unroll
                    for (int b = 0; b < 4; ++b) {
                        float2& s = sum[a][b];
                        s.x = fmaf(CONJ_Q ? v.y : -v.y, q[b].y, fmaf(v.x, q[b].x, s.x));
                        s.y = fmaf(CONJ_Q ? -v.x : v.x, q[b].y, fmaf(v.y, q[b].x, s.y));
                    }
                }
            }
        } else {
            const uint32_t st = frag + (uint32_t)(step % kPmStages) * STAGE;
            PmFragQ qr[MT], qi[MT];
#pragma unroll
            for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 v = pm_load8(st + (ROWS + 16 * mt + 8 * (i & 1)) * 64 + (i >> 1) * HALF);
                    pm_split(v.x, qr[mt].hi[i], qr[mt].lo[i]);
                    pm_split(v.y, qi[mt].hi[i], qi[mt].lo[i]);
                }
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                PmFragP pr, pi;
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const float2 v = pm_load8(st + nt * 512 + i * HALF);
                    pm_split(v.x, pr.hi[i], pr.lo[i]);
                    pm_split(v.y, pi.hi[i], pi.lo[i]);
                }
                const PmFragP n = pm_negated(CONJ_Q ? pr : pi);
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) pm_step<CONJ_Q, MODE == PM_FULL>(acc[nt][mt], qr[mt], qi[mt], pr, pi, n);
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();

    // results: line (i, j) of eight modes, the 8-byte modes permuted by a key of the line so that a half-warp (four j, four
    // pairs of i) covers all banks
    auto key = [](int i, int j) { return ((j >> 1) & 1) | (((i >> 1) & 3) << 1); };
    float2* out = reinterpret_cast<float2*>(smem_raw);
    if constexpr (MODE == PM_FMA) {
#pragma unroll
        for (int a = 0; a < 2 * NT; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const int i = row + 4 * a, j = col + b;
                out[(i * kPmCols + j) * kPmModes + (mode ^ key(i, j))] = make_float2(sum[a][b].x, CONJ_O ? -sum[a][b].y : sum[a][b].y);
            }
    } else {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int i = 8 * nt + 2 * t + (e & 1), j = 16 * mt + g + 8 * (e >> 1);
                    const PmSum& s = acc[nt][mt];
                    const float re = (e & 1) ? s.re[e >> 1].y : s.re[e >> 1].x, im = (e & 1) ? s.im[e >> 1].y : s.im[e >> 1].x;
                    out[(i * kPmCols + j) * kPmModes + (warp ^ key(i, j))] = make_float2(re, CONJ_O ? -im : im);
                }
    }
    __syncthreads();
    const long long m = m0 + 2 * (tid & 3);
    const float2 s0 = (m & 63) ? p.alpha : p.alpha0, s1 = p.alpha;       // m is even: m + 1 is no multiple of 64
#pragma unroll 2
    for (int line = tid >> 2; line < ROWS * kPmCols; line += kPmThreads / 4) {
        const int i = line / kPmCols, j = line % kPmCols, k = key(i, j);
        if (i0 + i >= p.I) break;
        const float4 v = *reinterpret_cast<const float4*>(out + line * kPmModes + 2 * ((tid & 3) ^ (k >> 1)));
        float2 a = (k & 1) ? make_float2(v.z, v.w) : make_float2(v.x, v.y), b = (k & 1) ? make_float2(v.x, v.y) : make_float2(v.z, v.w);
        if (p.splits > 1) {
            *reinterpret_cast<float4*>(p.partial + (((long long)split * p.I + i0 + i) * p.J + j0 + j) * p.modes + m) = make_float4(a.x, a.y, b.x, b.y);
            continue;
        }
        a = make_float2(s0.x * a.x - s0.y * a.y, s0.x * a.y + s0.y * a.x);
        b = make_float2(s1.x * b.x - s1.y * b.y, s1.x * b.y + s1.y * b.x);
        float2* o = p.o + (long long)(i0 + i) * p.o_si + (long long)(j0 + j) * p.o_sj + m * p.o_sm;
        if (p.o_vec) *reinterpret_cast<float4*>(o) = make_float4(a.x, a.y, b.x, b.y);
        else { o[0] = a; o[p.o_sm] = b; }
    }
}

// ---- gradient of weights that all modes share ----
//     partial[split, i, j] = conj( sum_r sum_m P[r, i, m] conj(Q[r, j, m]) ),  r = (b, m / 8)
// Here the sum runs along memory, so a matrix instruction is eight modes deep: lane 4 g + t takes modes 2 t and 2 t + 1 of
// its line (any assignment of modes to terms serves, as long as P and Q share it).  64 x 64 results per CTA, a warp
// 16 columns j by 32 rows i; the 64-byte pieces of odd lines change places in pairs, so that two adjacent lines at
// the same r cover all banks.
template <bool FULL>
__global__ void __launch_bounds__(kPmThreads, 2) cgemm_modesum_kernel(PerModeParams p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int iblocks = (p.I + kPmSumTile - 1) / kPmSumTile, jblocks = p.J / kPmSumTile;
    int item = blockIdx.x;
    const int i0 = (item % iblocks) * kPmSumTile; item /= iblocks;
    const int j0 = (item % jblocks) * kPmSumTile; item /= jblocks;
    const int split = item;
    const long long r0 = split * p.split_len;
    const long long r1 = (r0 + p.split_len < p.red) ? r0 + p.split_len : p.red;
    const int terms = r1 > r0 ? (int)(r1 - r0) : 0, steps = (terms + kPmSumTerms - 1) / kPmSumTerms;
    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(smem_raw);

    // copies: sixteen lanes bring the four terms of a line (256 bytes where the r are adjacent)
    const int c_line = tid >> 4, c_r = (tid >> 2) & 3, c_piece = tid & 3;
    const uint32_t c_dst = ring + (uint32_t)(c_line * 256 + ((c_r ^ (c_line & 1)) << 6) + (c_piece << 4));
    const float2* p_src = p.p + (r0 + c_r) * p.p_sr + (long long)(i0 + c_line) * p.p_si + 2 * c_piece;
    const float2* q_src = p.q + (r0 + c_r) * p.q_sr + (long long)(j0 + c_line) * p.q_sj + 2 * c_piece;
    auto fetch = [&](int step) {
        if (step < steps) {
            const uint32_t dst = c_dst + (uint32_t)(step % kPmStages) * kPmSumStageBytes;
            const bool live = step * kPmSumTerms + c_r < terms;
#pragma unroll
            for (int l = 0; l < kPmSumTile / 16; ++l) {
                const bool row = live && i0 + 16 * l + c_line < p.I;
                pm_copy16(dst + l * 4096, p_src + 16 * l * p.p_si, row);
                pm_copy16(dst + kPmSumTile * 256 + l * 4096, q_src + 16 * l * p.q_sj, live);
            }
            p_src += kPmSumTerms * p.p_sr;
            q_src += kPmSumTerms * p.q_sr;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    const int g = lane >> 2, t = lane & 3, iw = (warp & 1) * 32, jw = (warp >> 1) * 16;
    PmSum acc[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i] = PmSum{};
    follow_previous_kernel();
    admit_next_kernel();
#pragma unroll
    for (int s = 0; s < kPmStages - 1; ++s) fetch(s);
#pragma unroll 1
    for (int step = 0; step < steps; ++step) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kPmStages - 2) : "memory");
        __syncthreads();
        fetch(step + kPmStages - 1);
        const uint32_t st = ring + (uint32_t)(step % kPmStages) * kPmSumStageBytes + (uint32_t)(g * 256 + (t << 4));
#pragma unroll 2
        for (int r = 0; r < kPmSumTerms; ++r) {
            const uint32_t at = st + ((r ^ (g & 1)) << 6);
            const float4 q[2] = {pm_load16(at + (kPmSumTile + jw) * 256), pm_load16(at + (kPmSumTile + jw + 8) * 256)};
            PmFragQ qr, qi;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                pm_split(q[h].x, qr.hi[h], qr.lo[h]);
                pm_split(q[h].y, qi.hi[h], qi.lo[h]);
                pm_split(q[h].z, qr.hi[h + 2], qr.lo[h + 2]);
                pm_split(q[h].w, qi.hi[h + 2], qi.lo[h + 2]);
            }
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                const float4 v = pm_load16(at + (iw + 8 * nt) * 256);
                PmFragP pr, pi;
                pm_split(v.x, pr.hi[0], pr.lo[0]);
                pm_split(v.y, pi.hi[0], pi.lo[0]);
                pm_split(v.z, pr.hi[1], pr.lo[1]);
                pm_split(v.w, pi.hi[1], pi.lo[1]);
                pm_step<true, FULL>(acc[nt], qr, qi, pr, pi, pm_negated(pr));
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int i = i0 + iw + 8 * nt + 2 * t + (e & 1), j = j0 + jw + g + 8 * (e >> 1);
            const float2 re = acc[nt].re[e >> 1], im = acc[nt].im[e >> 1];
            if (i < p.I) p.partial[((long long)split * p.I + i) * p.J + j] = make_float2((e & 1) ? re.y : re.x, (e & 1) ? -im.y : -im.x);
        }
}

// adds the partial sums of the splits, in their order, and scales
__global__ void __launch_bounds__(256) permode_reduce_kernel(PerModeParams p) {
    const long long per = (long long)p.I * p.J * p.modes;
    follow_previous_kernel();
    admit_next_kernel();
    for (long long e = blockIdx.x * 256LL + threadIdx.x; e < per; e += gridDim.x * 256LL) {
        float2 v = make_float2(0.f, 0.f);
#pragma unroll 4
        for (int s = 0; s < p.splits; ++s) {
            const float2 t = p.partial[s * per + e];
            v.x += t.x; v.y += t.y;
        }
        const long long m = e % p.modes, ij = e / p.modes;
        const float2 s = (m & 63) ? p.alpha : p.alpha0;
        p.o[(ij / p.J) * p.o_si + (ij % p.J) * p.o_sj + m * p.o_sm] = make_float2(s.x * v.x - s.y * v.y, s.x * v.y + s.y * v.x);
    }
}
// The same for shared weights: few results (K x N) of many splits, so 32 threads share a result (a fixed order again).
constexpr int kPmSumReducers = 32;
__global__ void __launch_bounds__(32 * kPmSumReducers) modesum_reduce_kernel(PerModeParams p) {
    __shared__ float2 part[kPmSumReducers][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, per = p.I * p.J;
    const int e = blockIdx.x * 32 + lane;
    float2 v = make_float2(0.f, 0.f);
    follow_previous_kernel();
    admit_next_kernel();
    if (e < per) {
#pragma unroll 8
        for (int s = w; s < p.splits; s += kPmSumReducers) {
            const float2 t = p.partial[(long long)s * per + e];
            v.x += t.x; v.y += t.y;
        }
    }
    part[w][lane] = v;
    __syncthreads();
    if (w == 0 && e < per) {
#pragma unroll
        for (int i = 1; i < kPmSumReducers; ++i) { v.x += part[i][lane].x; v.y += part[i][lane].y; }
        p.o[(e / p.J) * p.o_si + (e % p.J) * p.o_sj] =
            make_float2(p.alpha.x * v.x - p.alpha.y * v.y, p.alpha.x * v.y + p.alpha.y * v.x);
    }
}

}  // namespace tfno
