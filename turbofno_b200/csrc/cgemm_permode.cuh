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
// README names as the FNO use case.  The operands are interleaved mode-fastest in memory, so the modes go
// on the LANES: a CTA takes eight adjacent modes (64 contiguous bytes of every row of P, Q and O), a warp
// 8 modes x 4 groups of TI rows i, and 8 columns j; eight warps cover 64 columns.  Slabs of P and Q for four r travel by 16-byte asynchronous copies through a ring
// of kPmStages.  FP32 FMA; a thread keeps TI x 8 complex sums, and per r its warp reads TI * 256 + 8 * 64 bytes
// of shared memory for TI * 32 FMA instructions.
//
// What bounds it (2D, 4096 modes, K = N = 64): up to 8 rows the 134 MB of weights (35 us at 1 row, 44 at 8; 20 us at
// copy speed); beyond that issue slots, 70 % used, 85 % of them FMA (16 rows 71 us, 32 rows 123 us; 30 and 60 us at the
// full FMA rate).  The four-modes-by-32-rows tile it replaces took 193 us at any batch up to 32.  Two CTAs per SM:
// one of 512 threads (32 rows) has nothing to cover its first loads and its stores with (137 us at 32 rows, 104
// against 92 at 20).  Packed two-wide FMAs take the same pipe cycles plus the moves that pair their operands
// (75 against 72 us at 16 rows).
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include "common.cuh"

namespace tfno {

constexpr int kPmModes = 8;            // adjacent modes per CTA
constexpr int kPmCols = 64;            // columns j per CTA: eight warps of 8
constexpr int kPmThreads = 4 * kPmCols;
constexpr int kPmSlab = 4;             // values of r per ring stage
constexpr int kPmStages = 4;

struct PerModeParams {
    int I, J;                          // J a multiple of 64
    long long red, modes;              // terms of the sum; modes: a multiple of 8
    const float2* p; long long p_sr, p_si;                 // P[r*p_sr + i*p_si + m]
    const float2* q; long long q_sr, q_sj, q_sm;           // Q[r*q_sr + j*q_sj + m*q_sm]
    float2* o; long long o_si, o_sj, o_sm;                 // O[i*o_si + j*o_sj + m*o_sm]
    float2* partial;                   // [splits][I][J][modes] (sum_modes: [splits][I][J]) when splits > 1 or sum_modes
    float2 alpha;
    float2 alpha0;                     // factor of the modes m % 64 == 0 (real fields: the ky = 0 column)
    int splits;                        // r is dealt to this many CTAs in runs of split_len
    long long split_len;
    int q_vec;                         // Q may be copied 16 bytes (two modes) at a time
};

// The launches (permode.cu).  `partial` must hold permode_partial_bytes() when that is not zero.
enum PermodeKind { PERMODE_APPLY, PERMODE_APPLY_CONJ, PERMODE_GRAD, PERMODE_GRAD_SHARED };
size_t permode_partial_bytes(const DeviceInfo& dev, const PerModeParams& p, PermodeKind kind);
int launch_permode(const DeviceInfo& dev, PerModeParams p, PermodeKind kind, cudaStream_t st);
// dst[k*N + n] = conj(w[k*sk + n*sn])
int launch_conjugate(const DeviceInfo& dev, const float2* w, long long sk, long long sn, int K, int N, float2* dst, cudaStream_t st);

template <int TI> __host__ __device__ constexpr size_t pm_stage_elems() { return (size_t)kPmSlab * (4 * TI + kPmCols) * kPmModes; }
template <int TI> __host__ __device__ constexpr size_t pm_smem_bytes() { return kPmStages * pm_stage_elems<TI>() * sizeof(float2); }

#if defined(__CUDACC__)
// copies `bytes` (16 or 8), or zeros when !live (the source is not read then)
__device__ __forceinline__ void pm_copy16(uint32_t dst, const void* src, bool live) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void pm_copy8(uint32_t dst, const void* src, bool live) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(live ? 8 : 0) : "memory");
}

// CONJ_Q: Q enters conjugated.  CONJ_O: the sum is conjugated before it is scaled (conj(P) Q = conj(P conj(Q))).
// SUM_MODES: the eight modes are added up; results go to `partial`.
template <int TI, bool CONJ_Q, bool CONJ_O, bool SUM_MODES>
__global__ void __launch_bounds__(kPmThreads, 2) cgemm_permode_kernel(PerModeParams p) {
    constexpr int THREADS = kPmThreads, ROWS = 4 * TI, LINES = ROWS + kPmCols;
    static_assert(4 * kPmSlab * ROWS <= THREADS && kPmSlab * kPmCols == THREADS, "a slab is one 16-byte piece of P and kPmSlab of Q per thread");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* ring = reinterpret_cast<float2*>(smem_raw);          // [stage][slab][ROWS + 64][8 modes]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m = lane & 7, ig = lane >> 3;
    const int wj = warp;
    // CTAs that differ only in their rows i are neighbours: they read the same Q, which is then served by the L2
    const int iblocks = (p.I + ROWS - 1) / ROWS, jblocks = p.J / kPmCols;
    long long item = blockIdx.x;
    const int i0 = (int)(item % iblocks) * ROWS; item /= iblocks;
    const int j0 = (int)(item % jblocks) * kPmCols; item /= jblocks;
    const int split = (int)(item % p.splits); item /= p.splits;
    const long long m0 = item * kPmModes;
    const long long r0 = split * p.split_len;
    const long long r1 = (r0 + p.split_len < p.red) ? r0 + p.split_len : p.red;
    const int slabs = r1 > r0 ? (int)((r1 - r0 + kPmSlab - 1) / kPmSlab) : 0;
    const uint32_t ring0 = (uint32_t)__cvta_generic_to_shared(ring);

    // A slab is 4 terms x (ROWS + 64) lines of four 16-byte pieces (two modes each).  Every thread keeps its
    // piece and line for good and one pointer per operand that moves on by a slab: the address arithmetic of a
    // fresh decomposition per copy took as many issue slots as the FMAs.
    const int piece = tid & 3;
    const int p_line = (tid >> 2) % ROWS, p_rr = (tid >> 2) / ROWS;         // p_rr < kPmSlab for tid < 16 * ROWS <= THREADS
    const bool p_row = p_rr < kPmSlab && i0 + p_line < p.I;
    const float2* p_src = p.p + (p_row ? (r0 + p_rr) * p.p_sr + (long long)(i0 + p_line) * p.p_si + m0 + 2 * piece : 0);
    const uint32_t p_dst = ring0 + (uint32_t)((p_rr * LINES + p_line) * kPmModes + 2 * piece) * 8u;
    const int q_line = tid >> 2;                                            // of all four terms
    const float2* q_src = p.q + r0 * p.q_sr + (long long)(j0 + q_line) * p.q_sj + m0 + 2 * piece;
    const uint32_t q_dst = ring0 + (uint32_t)((ROWS + q_line) * kPmModes + 2 * piece) * 8u;
    constexpr uint32_t STAGE = (uint32_t)(pm_stage_elems<TI>() * sizeof(float2));
    auto fetch = [&](int slab) {
        if (slab < slabs) {
            const uint32_t stage = (uint32_t)(slab % kPmStages) * STAGE;
            const int left = (int)(r1 - r0) - slab * kPmSlab;               // terms from this slab on
            if (p_rr < kPmSlab) pm_copy16(p_dst + stage, p_row && p_rr < left ? p_src : p.p, p_row && p_rr < left);
            p_src += p_row ? kPmSlab * p.p_sr : 0;
            if (p.q_vec) {
#pragma unroll
                for (int it = 0; it < kPmSlab; ++it) {
                    const bool live = it < left;
                    pm_copy16(q_dst + stage + (uint32_t)(it * LINES * kPmModes) * 8u, live ? q_src + it * p.q_sr : p.q, live);
                }
                q_src += kPmSlab * p.q_sr;
            } else {
                const long long rs = r0 + (long long)slab * kPmSlab;
#pragma unroll 1
                for (int i = tid; i < kPmSlab * kPmCols * 8; i += THREADS) {
                    const int mode = i & 7, line = (i >> 3) % kPmCols, rr = (i >> 3) / kPmCols;
                    const bool live = rr < left;
                    const float2* src = live ? p.q + (rs + rr) * p.q_sr + (long long)(j0 + line) * p.q_sj + (m0 + mode) * p.q_sm : p.q;
                    pm_copy8(ring0 + stage + (uint32_t)((rr * LINES + ROWS + line) * kPmModes + mode) * 8u, src, live);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    float2 acc[TI][8];
#pragma unroll
    for (int t = 0; t < TI; ++t)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[t][j] = make_float2(0.f, 0.f);
#pragma unroll
    for (int s = 0; s < kPmStages - 1; ++s) fetch(s);
    for (int slab = 0; slab < slabs; ++slab) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kPmStages - 2) : "memory");
        __syncthreads();                          // this slab has arrived; everybody has left the stage refilled next
        fetch(slab + kPmStages - 1);
        const float2* st = ring + (slab % kPmStages) * pm_stage_elems<TI>();
#pragma unroll
        for (int rr = 0; rr < kPmSlab; ++rr) {
            const float2* line = st + rr * LINES * kPmModes + m;
            float2 pv[TI];
#pragma unroll
            for (int t = 0; t < TI; ++t) pv[t] = line[(t * 4 + ig) * kPmModes];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float2 qv = line[(ROWS + wj * 8 + j) * kPmModes];
#pragma unroll
                for (int t = 0; t < TI; ++t) {
                    float2& a = acc[t][j];
                    if (CONJ_Q) {
                        a.x = fmaf(pv[t].x, qv.x, fmaf(pv[t].y, qv.y, a.x));
                        a.y = fmaf(pv[t].y, qv.x, fmaf(-pv[t].x, qv.y, a.y));
                    } else {
                        a.x = fmaf(pv[t].x, qv.x, fmaf(-pv[t].y, qv.y, a.x));
                        a.y = fmaf(pv[t].x, qv.y, fmaf(pv[t].y, qv.x, a.y));
                    }
                }
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");

#pragma unroll
    for (int t = 0; t < TI; ++t) {
        const int i = i0 + t * 4 + ig;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            float2 v = acc[t][j];
            if (CONJ_O) v.y = -v.y;
            if (SUM_MODES) {
#pragma unroll
                for (int d = 1; d < 8; d <<= 1) {
                    v.x += __shfl_xor_sync(0xffffffffu, v.x, d);
                    v.y += __shfl_xor_sync(0xffffffffu, v.y, d);
                }
                if (m == 0 && i < p.I) p.partial[((long long)split * p.I + i) * p.J + j0 + wj * 8 + j] = v;
            } else if (i < p.I) {
                if (p.splits > 1) p.partial[(((long long)split * p.I + i) * p.J + j0 + wj * 8 + j) * p.modes + m0 + m] = v;
                else {
                    const float2 s = ((m0 + m) & 63) ? p.alpha : p.alpha0;
                    p.o[(long long)i * p.o_si + (long long)(j0 + wj * 8 + j) * p.o_sj + (m0 + m) * p.o_sm] =
                        make_float2(s.x * v.x - s.y * v.y, s.x * v.y + s.y * v.x);
                }
            }
        }
    }
}

// adds the partial sums of the splits, in their order, and scales
template <bool SUM_MODES>
__global__ void __launch_bounds__(256) permode_reduce_kernel(PerModeParams p) {
    const long long per = (long long)p.I * p.J * (SUM_MODES ? 1 : p.modes);
    for (long long e = blockIdx.x * 256LL + threadIdx.x; e < per; e += gridDim.x * 256LL) {
        float2 v = make_float2(0.f, 0.f);
#pragma unroll 4
        for (int s = 0; s < p.splits; ++s) {
            const float2 t = p.partial[s * per + e];
            v.x += t.x; v.y += t.y;
        }
        const long long m = SUM_MODES ? 1 : e % p.modes, ij = SUM_MODES ? e : e / p.modes;
        const float2 s = (m & 63) ? p.alpha : p.alpha0;
        p.o[(ij / p.J) * p.o_si + (ij % p.J) * p.o_sj + (SUM_MODES ? 0 : m * p.o_sm)] = make_float2(s.x * v.x - s.y * v.y, s.x * v.y + s.y * v.x);
    }
}

#endif

}  // namespace tfno
