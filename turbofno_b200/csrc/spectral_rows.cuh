// Stand-alone transforms along the contiguous axis (fft_N_stride_DY / ifft_N_stride_DY of the reference, launches
// at fusion_variants/1D_A_exp_fft+cgemm+ifft/fused.cu:187-203).
#pragma once
#include "common.cuh"
#include "fft32.cuh"

namespace tfno {

// signal s -> element offset on the full-length side; 64-bit division is as dear as a tenth of a transform
TFNO_D long long row_offset(const RowsParams& p, long long s) {
    if (p.nsig <= 0x7fffffffLL) {
        const unsigned k = (unsigned)s / (unsigned)p.per_k;
        return (long long)((unsigned)s - k * (unsigned)p.per_k) * p.stride_row + (long long)k * p.stride_k;
    }
    return (s % p.per_k) * p.stride_row + (s / p.per_k) * p.stride_k;
}

// [signal][DY] -> compact [signal][64], DY = 64*RR.  On the 32-point transform (2*RR lanes per signal, 100 registers,
// 16 warps per SM): a warp loads, then computes, so what hides the loads is other warps.  With 64 samples per
// lane and eight warps 2^17 signals took 82.5 us at DY = 256 and 133.6 us at 512 (4.5 TB/s), here 62 and 103 us
// (5.9 TB/s); asking the L2 for the next signals (69 and 104 us on eight warps) adds nothing on sixteen.
template <int RR>
__global__ void __launch_bounds__(kThreads, 2) fft_rows_trunc_kernel(RowsParams p) {
    constexpr int R = 2 * RR, GROUPS = kThreads / R, PER = 64 / R;
    __shared__ __align__(16) float2 twF[R * 32];
    fill_forward_table32<R>(twF, threadIdx.x, kThreads);
    __syncthreads();
    const int g = threadIdx.x / R, r = threadIdx.x % R;
    const float2 coef = round1_coef32<R>(r);
    const long long nblk = (p.nsig + GROUPS - 1) / GROUPS;
    follow_previous_kernel();
    for (long long blk = blockIdx.x; blk < nblk; blk += gridDim.x) {
        if (gridDim.x >= nblk) admit_next_kernel();
        // clamp instead of branching so that every lane of a warp takes part in the shuffles
        long long s = blk * GROUPS + g;
        const bool live = s < p.nsig;
        if (!live) s = p.nsig - 1;
        const float2* row = p.in + row_offset(p, s) + r;
        float2 v[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = load_global(row + R * i);
        forward_trunc32<R>(v, twF, r, 1, coef);
        if (live) {
            float2* dst = p.out + s * kModes + PER * r;
#pragma unroll
            for (int j = 0; j < PER; j += 2)
                *reinterpret_cast<float4*>(dst + j) = make_float4(v[slot32(j)].x, v[slot32(j)].y, v[slot32(j + 1)].x, v[slot32(j + 1)].y);
        }
    }
}

// compact [signal][64] -> zero-padded inverse -> [signal][DY].  64 samples per lane: every lane reads all 64 modes of
// its signal, and half as many lanes read them.  Two CTAs of 128 threads instead of one of 256: 108 -> 104 us for 2^17
// signals of 512 samples (5.8 TB/s).
constexpr int kIfftRowsThreads = 128;
template <int R>
__global__ void __launch_bounds__(kIfftRowsThreads, 1) ifft_rows_pad_kernel(RowsParams p) {
    __shared__ __align__(16) float2 twI[R * 64];
    fill_inverse_table<R>(twI, threadIdx.x, kIfftRowsThreads, p.gain, p.conj_inverse != 0);
    __syncthreads();
    constexpr int GROUPS = kIfftRowsThreads / R;
    const int g = threadIdx.x / R, j1 = threadIdx.x % R;
    const long long nblk = (p.nsig + GROUPS - 1) / GROUPS;
    follow_previous_kernel();
    for (long long blk = blockIdx.x; blk < nblk; blk += gridDim.x) {
        if (gridDim.x >= nblk) admit_next_kernel();
        // clamp instead of branching so that every lane of a warp takes part in the store's shuffles
        long long s = blk * GROUPS + g;
        const bool live = s < p.nsig;
        if (!live) s = p.nsig - 1;
        float2 v[64];
        const float4* src = reinterpret_cast<const float4*>(p.in + s * kModes);
#pragma unroll
        for (int c = 0; c < 32; ++c) {
            const float4 q = load_global(src + c);
            v[2 * c] = make_float2(q.x, q.y);
            v[2 * c + 1] = make_float2(q.z, q.w);
        }
        if (p.conj_inverse) inverse_pad_lane<+1, R>(v, twI, j1);
        else inverse_pad_lane<-1, R>(v, twI, j1);
        store_decimated_paired<R>(v, p.out + row_offset(p, s), j1, live);
    }
}

}  // namespace tfno
