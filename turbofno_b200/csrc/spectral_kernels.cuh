// Hand-written sm_100a kernels of the spectral-convolution path (SIMT FP32 generation).
//
//   spectral_tile_kernel<R, FWD, INV>    one 64-mode row tile per CTA: [forward transform ->]
//                                        complex GEMM over channels [-> inverse transform]
//        <R,1,1>  fused FFT+CGEMM+iFFT   fusion_variants/1D_D_exp_fused_fft_cgemm_ifft/fused_fft_cgemm_ifft_7.cuh:9-222
//        <R,1,0>  fused FFT+CGEMM        fusion_variants/1D_B_exp_fused_fft_cgemm+ifft/fused_fft_cgemm_7.cuh:8-197
//        <R,0,1>  fused CGEMM+iFFT       fusion_variants/1D_C_exp_fft+fused_cgemm_ifft/fused_cgemm_ifft_7.cuh:9-222
//        <R,0,0>  CGEMM                  fusion_variants/1D_E_baseline/cgemm.cuh:4-205
//   fft_cols_trunc_kernel<R>, ifft_cols_pad_kernel<R>     strided-axis transforms
//        (fft_N_stride / ifft_N_stride, launches at fusion_variants/2D_D_exp_fused_fft_cgemm_ifft/fused_trunc_2D.cu:153-170)
//
// Unlike the reference's fused kernel, one CTA produces ALL N output channels of its row, so the
// forward transform of a row is never recomputed per N-tile (grid.y = N/64 in the reference).
#pragma once
#include "common.cuh"
#include "fft32.cuh"

namespace tfno {

constexpr int kSlabK = 8;          // channels per weight slab in the GEMM main loop
constexpr int kWPad = 2;           // row padding of the weight slab (bank spread for k-fastest fills)

// A [rows][64] complex tile in shared memory: 512-byte rows of 32 16-byte chunks.  The low three
// bits of the chunk index are XOR-swizzled so that (a) the R lanes of a group storing chunks
// 128*r bytes apart, (b) two adjacent rows written in the same phase, and (c) column reads that
// walk rows at a fixed chunk, all spread over distinct banks.
TFNO_HD int swz_chunk(int row, int c) {
    int x = ((((c >> 3) & 3) + ((row & 1) << 2)) ^ (((row >> 1) & 1) << 1)) & 7;
    return (c & ~7) | ((c & 7) ^ x);
}
// byte-free helpers: index in float2 units of element m of row `row`
TFNO_HD int tile_index(int row, int m) { return row * kModes + swz_chunk(row, m >> 1) * 2 + (m & 1); }

// The [n][64] tile handed from the GEMM to the inverse transform: chunk ^ (n & 7).
TFNO_HD int ctile_chunk(int n, int c) { return (c & ~7) | ((c & 7) ^ (n & 7)); }

struct TileParams {
    // problem
    long long rows;          // number of 64-mode row tiles: bs*dimX (1D), bs*64 (2D, per X-mode row)
    int K, N;
    // operand addressing, in complex elements
    const float2* x;         // FWD: signals; !FWD: compact spectrum A[m + k*M], M = rows*64
    long long x_stride_row;  // FWD: between rows
    long long x_stride_k;    // FWD: between channels
    const float2* w;
    long long w_stride_k, w_stride_n;
    float2* y;               // INV: signals out; !INV: compact C[m + n*M]
    long long y_stride_row, y_stride_n;
    float2 alpha, beta;      // beta only read when !INV
    float2 inv_gain;         // alpha * scale folded into the inverse twiddles (INV)
    int conj_inverse;        // 1: true inverse, 0: second forward transform
    int conj_w;              // !FWD && !INV: the weights enter conjugated
};

// After forward_trunc32<R>: lane r holds modes 64/R*r + j in v[slot32(j)].  Write them as 16-byte
// chunks into a swizzled tile row.
template <int R>
TFNO_D void store_modes_to_tile(const float2 (&v)[32], float2* tile, int row, int r) {
    constexpr int PER = 64 / R;
#pragma unroll
    for (int j = 0; j < PER; j += 2) {
        int m = PER * r + j;
        float4 q = make_float4(v[slot32(j)].x, v[slot32(j)].y, v[slot32(j + 1)].x, v[slot32(j + 1)].y);
        *reinterpret_cast<float4*>(tile + row * kModes + swz_chunk(row, m >> 1) * 2) = q;
    }
}

// ----------------------------------------------------------------------------------------------
// The row-tile kernel
// ----------------------------------------------------------------------------------------------
// The forward transform runs on the 32-point register FFT, L = 2 R = DY/32 lanes per signal: what counts here is the chain of
// one row, and a signal on twice the lanes is transformed in half the time while there are lanes to spare (8 channels of 128
// samples keep 32 of them busy, 32 channels of 256 all 256).  The inverse has N signals and stays on 64 samples per lane:
// its table for twice the lanes would take shared memory from the widest layers.  The first weights travel beside the
// forward transforms.  Calls back to back, us, with 64 samples per lane and now: 64 rows, 32 -> 128 channels, 256 samples 12.7 -> 12.0
// (where more channels leave no lanes to spare it can cost: 192 rows, 104 -> 64 channels 49.3 -> 50.3, of 512 samples 80.7 -> 73.9);
// together with launches that start beside the previous one's tail: 140 rows, 72 -> 64 channels 22.6 -> 19.4, 1200 rows, 200 -> 128 659 -> 610.
// The contraction alone (!FWD && !INV) of 64 output channels runs two CTAs per SM, which its 128 registers a thread just allow: 1024
// rows, 192 -> 64 channels 171 us, with 130 registers and one CTA 227.  Its weights are plain loads, which the compiler places
// among the multiplications (173 with loads in their order), and are conjugated on their way to shared memory: behind the load
// every slab waits for memory (256 -> 128 channels, 64 rows 32 against 39 us).
template <int R, bool FWD, bool INV, int NB>   // NB = N / 64
__global__ void __launch_bounds__(kThreads, !FWD && !INV && NB == 1 ? 2 : 1) spectral_tile_kernel(TileParams p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* sA = reinterpret_cast<float2*>(smem_raw);                 // [K][64] swizzled
    float2* sC = sA + (size_t)p.K * kModes;                            // [N][64] swizzled (INV only)
    float2* sW = sC + (INV ? (size_t)p.N * kModes : 0);                // [2][kSlabK][N]
    constexpr int L = 2 * R;                                           // lanes per signal, forward
    float2* twF = sW + 2 * kSlabK * (p.N + kWPad);                               // [L][32]
    float2* twI = twF + (FWD ? L * 32 : 0);                            // [R][64]

    const int tid = threadIdx.x;
    const int K = p.K, N = p.N;
    if (FWD) fill_forward_table32<L>(twF, tid, kThreads);
    if (INV) fill_inverse_table<R>(twI, tid, kThreads, p.inv_gain, p.conj_inverse != 0);
    __syncthreads();

    const long long M = p.rows * kModes;
    const int tm = tid & 15, tn = tid >> 4;        // GEMM thread tile: modes {2tm,2tm+1,32+2tm,33+2tm} x 4 n
    // blockIdx.y selects a block of N output channels: small batches of a wide layer are spread
    // over more CTAs that way (each repeats the row's forward transform, in parallel)
    const float2* wbase = p.w + (long long)blockIdx.y * N * p.w_stride_n;
    float2* ybase = p.y + (long long)blockIdx.y * N * (INV ? p.y_stride_n : M);

    constexpr int WPT = kSlabK * 64 * NB / kThreads;     // weight elements per thread per slab
    float2 wreg[WPT];
    auto fetch_slab = [&](int k0) {
#pragma unroll
        for (int i = 0; i < WPT; ++i) {
            int e = tid + i * kThreads;
            int kk, n;
            if (p.w_stride_n == 1) { n = e % N; kk = e / N; } else { kk = e % kSlabK; n = e / kSlabK; }
            const float2* src = wbase + (long long)(k0 + kk) * p.w_stride_k + (long long)n * p.w_stride_n;
            wreg[i] = (FWD || INV) ? load_global(src) : *src;
        }
    };
    auto stash_slab = [&](int buf) {
#pragma unroll
        for (int i = 0; i < WPT; ++i) {
            int e = tid + i * kThreads;
            int kk, n;
            if (p.w_stride_n == 1) { n = e % N; kk = e / N; } else { kk = e % kSlabK; n = e / kSlabK; }
            float2 v = wreg[i];
            if (!FWD && !INV && p.conj_w) v.y = -v.y;      // not in fetch_slab: it would wait for the load there
            sW[(buf * kSlabK + kk) * (N + kWPad) + n] = v;
        }
    };
    follow_previous_kernel();
    for (long long row = blockIdx.x; row < p.rows; row += gridDim.x) {
        if (gridDim.x >= p.rows) admit_next_kernel();
        fetch_slab(0);                                  // arrives beside the transforms
        // ---------------- stage 1: spectrum tile sA[k][m] ----------------
        if (FWD) {
            constexpr int GROUPS = kThreads / L;
            const int g = tid / L, r = tid % L;
            const int warp_g0 = (tid & ~31) / L;        // first group of this warp
            const float2 coef = round1_coef32<L>(r);
            for (int k0 = 0; k0 < K; k0 += GROUPS) {
                // Whole warps beyond K skip; inside a partly filled warp the spare lanes redo
                // channel K-1 so that every lane takes part in the shuffles of forward_trunc32.
                if (k0 + warp_g0 >= K) continue;
                const bool live = k0 + g < K;
                const int k = live ? k0 + g : K - 1;
                const float2* sig = p.x + row * p.x_stride_row + (long long)k * p.x_stride_k + r;
                float2 v[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) v[i] = load_global(sig + L * i);
                forward_trunc32<L>(v, twF, r, 1, coef);
                if (live) store_modes_to_tile<L>(v, sA, k, r);
            }
        } else {
            // compact spectrum: 64 consecutive m per channel; four loads on their way at a time
            for (int i0 = tid; i0 < K * 32; i0 += 4 * kThreads) {
                float4 q[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int i = i0 + j * kThreads;
                    if (i < K * 32) q[j] = load_global(reinterpret_cast<const float4*>(p.x + row * kModes + (long long)(i >> 5) * M) + (i & 31));
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int i = i0 + j * kThreads, k = i >> 5;
                    if (i < K * 32) *reinterpret_cast<float4*>(sA + k * kModes + swz_chunk(k, i & 31) * 2) = q[j];
                }
            }
        }

        // ---------------- stage 2: C[m][n] = sum_k A[k][m] W[k][n] ----------------
        float2 acc[NB][4][4];
#pragma unroll
        for (int b = 0; b < NB; ++b)
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[b][i][j] = make_float2(0.f, 0.f);

        stash_slab(0);
        __syncthreads();   // sA complete, slab 0 visible

        for (int k0 = 0, buf = 0; k0 < K; k0 += kSlabK, buf ^= 1) {
            const bool more = k0 + kSlabK < K;
            if (more) fetch_slab(k0 + kSlabK);
#pragma unroll
            for (int kk = 0; kk < kSlabK; ++kk) {
                const int k = k0 + kk;
                const float4 a01 = *reinterpret_cast<const float4*>(sA + k * kModes + swz_chunk(k, tm) * 2);
                const float4 a23 = *reinterpret_cast<const float4*>(sA + k * kModes + swz_chunk(k, 16 + tm) * 2);
                const float2 a[4] = {make_float2(a01.x, a01.y), make_float2(a01.z, a01.w),
                                     make_float2(a23.x, a23.y), make_float2(a23.z, a23.w)};
#pragma unroll
                for (int b = 0; b < NB; ++b) {
                    const float4* wp = reinterpret_cast<const float4*>(sW + (buf * kSlabK + kk) * (N + kWPad) + 64 * b + 4 * tn);
                    const float4 w01 = wp[0], w23 = wp[1];
                    const float2 w[4] = {make_float2(w01.x, w01.y), make_float2(w01.z, w01.w),
                                         make_float2(w23.x, w23.y), make_float2(w23.z, w23.w)};
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            acc[b][i][j].x = fmaf(a[i].x, w[j].x, acc[b][i][j].x);
                            acc[b][i][j].x = fmaf(-a[i].y, w[j].y, acc[b][i][j].x);
                            acc[b][i][j].y = fmaf(a[i].x, w[j].y, acc[b][i][j].y);
                            acc[b][i][j].y = fmaf(a[i].y, w[j].x, acc[b][i][j].y);
                        }
                }
            }
            if (more) stash_slab(buf ^ 1);
            __syncthreads();
        }

        // ---------------- stage 3: epilogue ----------------
        if (INV) {
            // alpha and the 1/DY scale live in the inverse twiddles; hand C to the transform lanes
#pragma unroll
            for (int b = 0; b < NB; ++b)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int n = 64 * b + 4 * tn + j;
                    float4 q0 = make_float4(acc[b][0][j].x, acc[b][0][j].y, acc[b][1][j].x, acc[b][1][j].y);
                    float4 q1 = make_float4(acc[b][2][j].x, acc[b][2][j].y, acc[b][3][j].x, acc[b][3][j].y);
                    *reinterpret_cast<float4*>(sC + n * kModes + ctile_chunk(n, tm) * 2) = q0;
                    *reinterpret_cast<float4*>(sC + n * kModes + ctile_chunk(n, 16 + tm) * 2) = q1;
                }
            __syncthreads();
            constexpr int GROUPS = kThreads / R;
            const int g = tid / R, j1 = tid % R;
            for (int n0 = 0; n0 < N; n0 += GROUPS) {
                int n = n0 + g;
                if (n < N) {
                    float2 v[64];
#pragma unroll
                    for (int c = 0; c < 32; ++c) {
                        float4 q = *reinterpret_cast<const float4*>(sC + n * kModes + ctile_chunk(n, c) * 2);
                        v[2 * c] = make_float2(q.x, q.y);
                        v[2 * c + 1] = make_float2(q.z, q.w);
                    }
                    if (p.conj_inverse) inverse_pad_lane<+1, R>(v, twI, j1);
                    else inverse_pad_lane<-1, R>(v, twI, j1);
                    store_decimated_paired<R>(v, ybase + row * p.y_stride_row + (long long)n * p.y_stride_n, j1);   // whole warps: N is a multiple of 64
                }
            }
            __syncthreads();   // sC and sA are rewritten by the next row
        } else {
            const bool use_beta = (p.beta.x != 0.f || p.beta.y != 0.f);
#pragma unroll
            for (int b = 0; b < NB; ++b)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int n = 64 * b + 4 * tn + j;
                    float2* dst = ybase + row * kModes + (long long)n * M;
                    float2 o[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) o[i] = cmul(acc[b][i][j], p.alpha);
                    float4* d0 = reinterpret_cast<float4*>(dst + 2 * tm);
                    float4* d1 = reinterpret_cast<float4*>(dst + 32 + 2 * tm);
                    if (use_beta) {
                        float4 c0 = *d0, c1 = *d1;
                        o[0] = cadd(o[0], cmul(make_float2(c0.x, c0.y), p.beta));
                        o[1] = cadd(o[1], cmul(make_float2(c0.z, c0.w), p.beta));
                        o[2] = cadd(o[2], cmul(make_float2(c1.x, c1.y), p.beta));
                        o[3] = cadd(o[3], cmul(make_float2(c1.z, c1.w), p.beta));
                    }
                    *d0 = make_float4(o[0].x, o[0].y, o[1].x, o[1].y);
                    *d1 = make_float4(o[2].x, o[2].y, o[3].x, o[3].y);
                }
            __syncthreads();   // sA is rewritten by the next row
        }
    }
}

// ----------------------------------------------------------------------------------------------
// Stand-alone transforms along the strided (X) axis of [image][DX][DY] data
// ----------------------------------------------------------------------------------------------
struct ColsParams {
    long long nimg;
    long long per_k;           // images per channel: image i -> channel i / per_k, batch i % per_k
    int DY;                    // row length = element stride along X
    const float2* in;
    float2* out;
    long long stride_b, stride_k;   // image strides of the full-size side; the 64-row side is compact
    float2 gain;
    int conj_inverse;
};

// [img][DX][DY] -> [img][64][DY]   (DX = 64*R)
template <int R>
__global__ void __launch_bounds__(kThreads, 1) fft_cols_trunc_kernel(ColsParams p) {
    __shared__ __align__(16) float2 twF[R * 64];
    fill_forward_table<R>(twF, threadIdx.x, kThreads);
    __syncthreads();
    constexpr int GROUPS = kThreads / R, PER = 64 / R;
    const int g = threadIdx.x / R, r = threadIdx.x % R;
    const long long ncol = p.nimg * p.DY;
    const long long nblk = (ncol + GROUPS - 1) / GROUPS;
    follow_previous_kernel();
    for (long long blk = blockIdx.x; blk < nblk; blk += gridDim.x) {
        if (gridDim.x >= nblk) admit_next_kernel();
        long long c = blk * GROUPS + g;
        const bool live = c < ncol;
        if (!live) c = ncol - 1;
        const long long img = c / p.DY;
        const int col = (int)(c % p.DY);
        float2 v[64];
        load_decimated<R>(v, p.in + (img % p.per_k) * p.stride_b + (img / p.per_k) * p.stride_k + col, p.DY, r);
        forward_trunc<R>(v, twF, r);
        if (live) {
            float2* dst = p.out + img * (long long)kModes * p.DY + col;
#pragma unroll
            for (int j = 0; j < PER; ++j) dst[(long long)(PER * r + j) * p.DY] = v[slot(j)];
        }
    }
}

// [img][64][DY] -> zero-pad rows -> inverse along X -> [img][DX][DY]
template <int R>
__global__ void __launch_bounds__(kThreads, 1) ifft_cols_pad_kernel(ColsParams p) {
    __shared__ __align__(16) float2 twI[R * 64];
    fill_inverse_table<R>(twI, threadIdx.x, kThreads, p.gain, p.conj_inverse != 0);
    __syncthreads();
    constexpr int GROUPS = kThreads / R;
    const int g = threadIdx.x / R, j1 = threadIdx.x % R;
    const long long ncol = p.nimg * p.DY;
    const long long nblk = (ncol + GROUPS - 1) / GROUPS;
    follow_previous_kernel();
    for (long long blk = blockIdx.x; blk < nblk; blk += gridDim.x) {
        if (gridDim.x >= nblk) admit_next_kernel();
        long long c = blk * GROUPS + g;
        if (c >= ncol) continue;
        const long long img = c / p.DY;
        const int col = (int)(c % p.DY);
        float2 v[64];
        const float2* src = p.in + img * (long long)kModes * p.DY + col;
#pragma unroll
        for (int m = 0; m < 64; ++m) v[m] = load_global(src + (long long)m * p.DY);
        if (p.conj_inverse) inverse_pad_lane<+1, R>(v, twI, j1);
        else inverse_pad_lane<-1, R>(v, twI, j1);
        store_decimated<R>(v, p.out + (img % p.per_k) * p.stride_b + (img / p.per_k) * p.stride_k + col, p.DY, j1);
    }
}

// ----------------------------------------------------------------------------------------------
// Data-movement kernels of the library (cuFFT + cuBLAS) pipeline: keep the first 64 of DY
// entries of each signal / zero-fill back (fusion_variants/1D_E_baseline/fused.cu:13-63), and
// the corner-block forms for images (fusion_variants/2D_E_baseline/fused_trunc_2D.cu:13-71).
// One float4 = two complex per thread, grid-stride.
// ----------------------------------------------------------------------------------------------
__global__ void truncate_rows_kernel(const float4* __restrict__ in, float4* __restrict__ out,
                                     long long nsig, int DY) {
    const long long total = nsig * 32;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        long long s = i >> 5; int c = (int)(i & 31);
        out[i] = __ldg(in + s * (DY / 2) + c);
    }
}
__global__ void zero_pad_rows_kernel(const float4* __restrict__ in, float4* __restrict__ out,
                                     long long nsig, int DY) {
    const int per = DY / 2;
    const long long total = nsig * per;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        long long s = i / per; int c = (int)(i % per);
        out[i] = c < 32 ? __ldg(in + s * 32 + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
}
__global__ void truncate_corner_kernel(const float4* __restrict__ in, float4* __restrict__ out,
                                       long long nimg, int DX, int DY) {
    const long long total = nimg * 64 * 32;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        int c = (int)(i & 31); long long t = i >> 5; int x = (int)(t & 63); long long img = t >> 6;
        out[i] = __ldg(in + (img * DX + x) * (DY / 2) + c);
    }
}
__global__ void zero_pad_corner_kernel(const float4* __restrict__ in, float4* __restrict__ out,
                                       long long nimg, int DX, int DY) {
    const int per = DY / 2;
    const long long total = nimg * DX * per;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        int c = (int)(i % per); long long t = i / per; int x = (int)(t % DX); long long img = t / DX;
        out[i] = (c < 32 && x < 64) ? __ldg(in + (img * 64 + x) * 32 + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

}  // namespace tfno
