// Whole-image 2-D transforms on the 32-point register FFT (fft32.cuh): the image is cut into parts of
// 64 rows that small CTAs of 128 threads (or two parts, 256 threads) work on, so that four (two) CTAs
// share an SM and one's DRAM phase overlaps the others' arithmetic, and a single image still occupies
// several SMs.  No counterpart in the reference, which round-trips the X-transformed image through
// global memory (fusion_variants/2D_D_exp_fused_fft_cgemm_ifft/fused_trunc_2D.cu:188-192).
//
//   forward  a cluster of DX/64 CTAs per image.  Each transforms 64 rows along Y and scatters the kept
//            columns through distributed shared memory: CTA c of the cluster collects columns
//            c*64/C .. of ALL rows (32 KB), then transforms them along X.  A cluster takes ONE image: a
//            cluster barrier says that the peers run before the first remote store (the row loads and
//            transforms hide it), a second one separates the passes.  With many images (C = 1) a CTA
//            takes one after the other.
//   inverse  no exchange at all: lane j1 of the zero-padded X transform produces exactly the image
//            rows RX*j2 + j1, so a CTA takes CLS of the RX residue classes, transforms the 64 columns
//            for those rows only (every part re-reads the 32 KB spectrum, from the L2), then its rows.
//
// REAL: the full-size side holds real samples.  Two rows share one complex transform (fft_real.cuh), whose lanes own each kept
// mode together with its mirror image: 2 Re(ifft2(Z')) with the ky = 0 column entering once.
#pragma once
#include "fft_real.cuh"
#include <type_traits>
#include "common.cuh"

namespace tfno {

// ---- shared-memory tiles ----
// inverse: [rows][64] complex, 512-byte rows of 32 16-byte chunks, low three bits XOR-ed with `key`, the number of
// the row (of the pair of rows): the groups of a warp read adjacent rows (pairs) at the same chunk.  Local row i is
// image row RX*(i/CLS) + part*CLS + i%CLS, so that a round writes runs of adjacent image rows.
TFNO_HD int rtile_chunk(int key, int c) { return (c & ~7) | ((c ^ key) & 7); }
// forward: [DX rows][64/C columns] complex, rows of 32/C 16-byte chunks, low three bits XOR-ed with a number
// of the row and (C = 1) of the chunk's group of eight.  The X pass reads RX adjacent rows at one pair (RX = 8)
// or quadruple (RX = 4) of chunks: the plain row number spreads the former over the banks, the row number
// rotated by one bit the latter.  REAL and RX = 4: the lanes store two or four adjacent chunks of every second row.
template <int RX, int C, bool REAL>
TFNO_HD int xtile_index(int row, int col) {
    const int c = col >> 1;
    const int s = ((RX == 8) ? (row & 7) : REAL ? ((((row >> 2) ^ row) & 1) << 2) | (row & 2) : (((row & 1) << 2) | ((row >> 1) & 3))) ^
                  (C == 1 ? (c >> 3) & 3 : 0);
    return row * (64 / C) + (((c & ~7) | ((c ^ s) & 7)) << 1) + (col & 1);
}
// REAL: the inverse reads two or four adjacent chunks of every second row
TFNO_HD int rtile_pair_key(int pair) { return ((pair & 1) << 2) | (pair & 2) | ((pair >> 2) & 1); }
template <int RX, int RY, int C, bool REAL> inline constexpr size_t fwd_image_smem_bytes() {
    return (size_t)(32 * RX * (64 / C) + RX * 32 + (REAL ? RY * 16 + 8 * (64 * RX / C) : RY == 8 ? kTable256 + 64 * (8 * RX / C) : RY * 32)) * sizeof(float2);
}
template <int RY, int CLS> inline constexpr size_t inv64_image_smem_bytes() {
    return (size_t)(64 * CLS * kModes + RY * 64 + CLS * 64) * sizeof(float2);
}
template <int RY, int CLS, bool REAL> inline constexpr size_t inv_image_smem_bytes() {
    return (size_t)(32 * CLS * kModes + RY * 32 + CLS * 32 + (REAL ? 8 * (64 * CLS) : 0)) * sizeof(float2);
}

#if defined(__CUDACC__)
TFNO_D uint32_t shared_address(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
TFNO_D uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
TFNO_D uint32_t map_to_rank(uint32_t addr, uint32_t rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    return a;
}
TFNO_D void store_cluster16(uint32_t addr, float2 a, float2 b) {
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y) : "memory");
}
TFNO_D void store_cluster8(uint32_t addr, float2 a) { asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(a.x), "f"(a.y) : "memory"); }
TFNO_D void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
TFNO_D void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// ------------------------------------------------------------------------------------------
// [image][DX][DY] -> [image][64][64]      RX = DX/32, RY = DY/32 (4 or 8 each)
// ------------------------------------------------------------------------------------------
template <int RX, int RY, int C, bool REAL>
__global__ void __launch_bounds__(64 * RX / C, 8 * C / RX) fft2d_trunc_kernel(ImageParams p) {
    constexpr int T = 64 * RX / C, COLS = 64 / C, DX = 32 * RX, DY = 32 * RY, ROWS = DX / C, PERY = 64 / RY, PERX = 64 / RX;
    using Sample = typename std::conditional<REAL, float, float2>::type;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* sX = reinterpret_cast<float2*>(smem_raw);           // [DX][COLS] swizzled: this CTA's columns
    constexpr bool ONCE = RY == 8;                               // rows of 256 samples: one exchange (fft256.cuh)
    float2* twX = sX + DX * COLS;                                // [RX][32]
    float2* twY = twX + RX * 32;                                 // factors of the rows, then the exchanged values of the groups of lanes
    const int tid = threadIdx.x;
    const int rank = C > 1 ? (int)cluster_rank() : 0;
    if constexpr (REAL) fill_real_table<DY>(twY, tid, T);
    else if constexpr (ONCE) fill_table256(twY, tid, T);
    else fill_forward_table32<RY>(twY, tid, T);
    fill_forward_table32<RX>(twX, tid, T, p.centered_x != 0);
    __syncthreads();
    if constexpr (REAL) {                                        // the 1/2 of the separated rows
        for (int i = tid; i < RX * 32; i += T) twX[i] = make_float2(0.5f * twX[i].x, 0.5f * twX[i].y);
        __syncthreads();
    }
    const int g = tid / RY, r = tid % RY;
    const float2 coefY = round1_coef32<RY>(r);
    const int col = tid / RX, rx = tid % RX;
    const float2 coefX = round1_coef32<RX>(rx);
    // modes m, m + 1 (or m alone) of image row `row`: to the CTA of the cluster that collects their columns
    auto put = [&](int row, int m, float2 a, float2 b) {
        const int at = xtile_index<RX, C, REAL>(row, m % COLS);
        if constexpr (C > 1) store_cluster16(map_to_rank(shared_address(sX), (uint32_t)(m / COLS)) + 8u * (uint32_t)at, a, b);
        else *reinterpret_cast<float4*>(sX + at) = make_float4(a.x, a.y, b.x, b.y);
    };
    auto put1 = [&](int row, int m, float2 a) {
        const int at = xtile_index<RX, C, REAL>(row, m % COLS);
        if constexpr (C > 1) store_cluster8(map_to_rank(shared_address(sX), (uint32_t)(m / COLS)) + 8u * (uint32_t)at, a);
        else sX[at] = a;
    };
    constexpr int GROUPS = T / RY, LINES = REAL ? 2 : 1, STEP = GROUPS * LINES, ROUNDS = ROWS / STEP;
    static_assert(ROUNDS >= 1, "a round of row transforms fits the CTA's rows");
    const long long step = C > 1 ? p.nimg : gridDim.x;           // a cluster's only image; there are as many clusters as images
    auto rows_of = [&](long long img) {
        return reinterpret_cast<const Sample*>(p.in) + (img % p.per_k) * p.stride_b + (img / p.per_k) * p.stride_k + (long long)rank * ROWS * DY;
    };
    if constexpr (C > 1) cluster_arrive();                       // this CTA runs: its shared memory may be written
    follow_previous_kernel();
    for (long long img = blockIdx.x / C; img < p.nimg; img += step) {
        if (step >= p.nimg) admit_next_kernel();
        const Sample* src = rows_of(img);
        const Sample* next = C == 1 && img + step < p.nimg ? rows_of(img + step) : nullptr;
#pragma unroll 1
        for (int i0 = 0; i0 < ROUNDS; ++i0) {
            // REAL, four groups to a warp: the two of a half-warp take pairs of rows that lie two apart (bank conflicts of put1)
            const int x = i0 * STEP + (REAL && RY == 8 ? (g & ~3) | ((g & 1) << 1) | ((g >> 1) & 1) : g) * LINES;
            const int gx = rank * ROWS + x;
            float2 v[32];
            float2 (&v0)[16] = *reinterpret_cast<float2(*)[16]>(&v[0]), (&v1)[16] = *reinterpret_cast<float2(*)[16]>(&v[16]);
            if constexpr (REAL) {
                constexpr int Q = RealRows<DY>::Q, K1 = RealRows<DY>::K1;
                const Sample* row = src + (long long)x * DY + Q * r;
                auto load2 = [&](int q, int j) {                       // samples q, q + 1 of both rows
                    const float2 a = load_global(reinterpret_cast<const float2*>(row + 16 * j + q)), b = load_global(reinterpret_cast<const float2*>(row + DY + 16 * j + q));
                    v[q * K1 + j] = make_float2(a.x, b.x);
                    v[(q + 1) * K1 + j] = make_float2(a.y, b.y);
                };
                if (Q == 2 || !p.rows16) {
#pragma unroll
                    for (int j = 0; j < K1; ++j)
#pragma unroll
                        for (int q = 0; q < Q; q += 2) load2(q, j);
                } else if constexpr (Q == 4) {
#pragma unroll
                    for (int j = 0; j < K1; ++j) {
                        const float4 a = load_global(reinterpret_cast<const float4*>(row + 16 * j)), b = load_global(reinterpret_cast<const float4*>(row + DY + 16 * j));
                        v[j] = make_float2(a.x, b.x);
                        v[K1 + j] = make_float2(a.y, b.y);
                        v[2 * K1 + j] = make_float2(a.z, b.z);
                        v[3 * K1 + j] = make_float2(a.w, b.w);
                    }
                }
            } else if constexpr (ONCE) {
                const float4* row = reinterpret_cast<const float4*>(src + (long long)x * DY) + r;
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float4 q = load_global(row + 8 * i);
                    v0[i] = make_float2(q.x, q.y);
                    v1[i] = make_float2(q.z, q.w);
                }
            } else {
                const Sample* row = src + (long long)x * DY + r;
#pragma unroll
                for (int i = 0; i < 32; ++i) v[i] = load_global(row + RY * i);
            }
            // The rows of the next round (this image's or the next one's) travel to the L2 meanwhile.  Two rounds
            // ahead is slower: 913 against 880 us for 8192 images of 256 x 256 (rows on the 32-point transform).
            const Sample* ahead = i0 + 1 < ROUNDS ? src + (long long)(i0 + 1) * STEP * DY : next;
            if (ahead) prefetch_l2_block(ahead, STEP * DY * (int)sizeof(Sample), tid, T);
            if constexpr (REAL) {
                constexpr int N = DY, Q = RealRows<N>::Q, K1 = RealRows<N>::K1, M = RealRows<N>::M;
                float2 fa[16], fb[16];
                real_forward<N>(*reinterpret_cast<float2(*)[Q][K1]>(&v[0]), twY, twY + N / 2 + RealRows<N>::SCRATCH * g, r, g & 1, fa, fb);
                if (C > 1 && i0 == 0) cluster_wait();
                const int kb = real_mode<N>(1, r);
#pragma unroll
                for (int k2 = 0; k2 < M; ++k2)
#pragma unroll
                    for (int part = 0; part < 2; ++part) {
                        float2 a, b;
                        real_separate<N>(fa, fb, part, r == 0, k2, a, b);
                        put1(gx, (part ? kb : r) + K1 * k2, a);
                        put1(gx + 1, (part ? kb : r) + K1 * k2, b);
                    }
            } else if constexpr (ONCE) {
                fft16<-1>(v0);
                fft16<-1>(v1);
                float2* scratch = twY + kTable256 + 64 * g;
                float2 out[2][4];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    float2 f[16];
#pragma unroll
                    for (int q = 0; q < 2; ++q) exchange256(scratch, r, g & 1, q, f, [&](int d) { return (q ? v1 : v0)[slot16(2 * d + e)]; });
                    combine256(f, twY, 2 * r + e, out[e]);
                }
                if (C > 1 && i0 == 0) cluster_wait();
#pragma unroll
                for (int k2 = 0; k2 < 4; ++k2) put(gx, 2 * r + 16 * k2, out[0][k2], out[1][k2]);
            } else {
                forward_trunc32<RY>(v, twY, r, 1, coefY);
                if (C > 1 && i0 == 0) cluster_wait();
#pragma unroll
                for (int j = 0; j < PERY; j += 2) put(gx, PERY * r + j, v[slot32(j)], v[slot32(j + 1)]);
            }
        }
        if constexpr (C > 1) { cluster_arrive(); cluster_wait(); }
        else __syncthreads();
        {
            float2 v[32];
#pragma unroll
            for (int n = 0; n < 32; ++n) v[n] = sX[xtile_index<RX, C, REAL>(RX * n + rx, col)];
            if constexpr (C == 1) __syncthreads();              // columns read: the next image may be stored
            forward_trunc32<RX>(v, twX, rx, 1, coefX);
            float2* dst = p.out + img * (long long)(kModes * kModes) + rank * COLS + col;
#pragma unroll
            for (int j = 0; j < PERX; ++j) dst[(PERX * rx + j) * kModes] = v[slot32(j)];
        }
    }
}

// ------------------------------------------------------------------------------------------
// [image][64][64] -> zero-pad -> inverse along X into shared memory -> inverse along Y -> [image][DX][DY]
// INVERSE: true inverse or a second forward transform.
// ------------------------------------------------------------------------------------------
template <int RX, int RY, int CLS, bool INVERSE, bool REAL>
__global__ void __launch_bounds__(64 * CLS, 8 / CLS) ifft2d_pad_kernel(ImageParams p) {
    static_assert(INVERSE || !REAL, "a real field has a true inverse only");
    constexpr int T = 64 * CLS, ROWS = 32 * CLS, PARTS = RX / CLS, DY = 32 * RY, SIGN = INVERSE ? 1 : -1;
    constexpr int GROUPS = T / RY, LINES = REAL ? 2 : 1;
    using Sample = typename std::conditional<REAL, float, float2>::type;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* sY = reinterpret_cast<float2*>(smem_raw);           // [ROWS][64] swizzled
    float2* twY = sY + ROWS * kModes;                            // [RY][32]
    float2* twX = twY + RY * 32;                                 // [CLS][32]; REAL: then the exchanged values of the groups of lanes
    const int tid = threadIdx.x;
    const int part = blockIdx.x % PARTS;                         // the grid is a multiple of PARTS
    if constexpr (REAL) fill_real_table<DY>(twY, tid, T);
    else fill_inverse_table32_folded<RY>(twY, tid, T, make_float2(1.f, 0.f), INVERSE);
    for (int i = tid; i < CLS * 32; i += T) {                    // rows part*CLS .. of fill_inverse_table32_folded<RX>
        const int j1 = part * CLS + (i >> 5), m = i & 31;        // modes -32..31: times e^{-2 pi i j1 / RX}
        const int e = (INVERSE && p.centered_x) ? (j1 * m - 32 * j1) & (32 * RX - 1) : (j1 * m) & (32 * RX - 1);
        twX[i] = cmul(p.gain, unit_root(e, 32 * RX, INVERSE ? 1.0f : -1.0f));
    }
    __syncthreads();
    const int ky = tid & 63, jl = tid >> 6;
    const float2 coefX = inverse_fold_coef32<RX>(part * CLS + jl, INVERSE);
    const int g = tid / RY, j1 = tid % RY;
    const float2 coefY = inverse_fold_coef32<RY>(j1, INVERSE);
    const bool odd = (j1 & 1) != 0;
    follow_previous_kernel();
    for (long long img = blockIdx.x / PARTS; img < p.nimg; img += gridDim.x / PARTS) {
        if (gridDim.x / PARTS >= p.nimg) admit_next_kernel();
        const float2* src = p.in + img * (long long)(kModes * kModes) + ky;
        Sample* dst = reinterpret_cast<Sample*>(p.out) + (img % p.per_k) * p.stride_b + (img / p.per_k) * p.stride_k;
        {
            float2 v[32];
#pragma unroll
            for (int m = 0; m < 32; m += 2) {
                const float4 t = *reinterpret_cast<const float4*>(twX + jl * 32 + m);
                v[m] = cmul(cmadd(load_global(src + m * kModes), coefX, load_global(src + (m + 32) * kModes)), make_float2(t.x, t.y));
                v[m + 1] = cmul(cmadd(load_global(src + (m + 1) * kModes), coefX, load_global(src + (m + 33) * kModes)), make_float2(t.z, t.w));
            }
            fft32<SIGN>(v);
#pragma unroll
            for (int j2 = 0; j2 < 32; ++j2) {
                const int row = j2 * CLS + jl;
                sY[row * kModes + rtile_chunk(REAL ? rtile_pair_key(row / 2) : row, ky >> 1) * 2 + (ky & 1)] = v[slot32(j2)];
            }
        }
        __syncthreads();
        // folded input of lane j1, modes 2c and 2c + 1: u[m] = T[m] (C[m] + coef C[m + 32])
        auto folded = [&](const float2* line, int key, int c, float2& u0, float2& u1) {
            const float4 lo = *reinterpret_cast<const float4*>(line + rtile_chunk(key, c) * 2);
            const float4 hi = *reinterpret_cast<const float4*>(line + rtile_chunk(key, c + 16) * 2);
            const float4 t = *reinterpret_cast<const float4*>(twY + tw_index<RY>(j1, 2 * c));
            u0 = cmul(cmadd(make_float2(lo.x, lo.y), coefY, make_float2(hi.x, hi.y)), make_float2(t.x, t.y));
            u1 = cmul(cmadd(make_float2(lo.z, lo.w), coefY, make_float2(hi.z, hi.w)), make_float2(t.z, t.w));
        };
#pragma unroll 1
        for (int x0 = 0; x0 < ROWS; x0 += GROUPS * LINES) {
            const int lr = x0 + g * LINES;
            const int x = RX * (lr / CLS) + part * CLS + lr % CLS;       // image row of local row lr (REAL: the next one is x + 1)
            if constexpr (REAL) {
                constexpr int N = DY, Q = RealRows<N>::Q, K1 = RealRows<N>::K1, M = RealRows<N>::M;
                const int key = rtile_pair_key(lr / 2), kb = real_mode<N>(1, j1);
                const float2 *la = sY + lr * kModes, *lb = la + kModes;
                float2 aA[M], bA[M], aB[M], bB[M], fa[16], fb[16], v[Q][K1];
#pragma unroll
                for (int k2 = 0; k2 < M; ++k2) {
                    const int ka = j1 + K1 * k2, kk = kb + K1 * k2;
                    const int atA = rtile_chunk(key, ka >> 1) * 2 + (ka & 1), atB = rtile_chunk(key, kk >> 1) * 2 + (kk & 1);
                    aA[k2] = la[atA]; bA[k2] = lb[atA];
                    aB[k2] = la[atB]; bB[k2] = lb[atB];
                }
                real_join<N>(fa, fb, aA, bA, aB, bB, j1 == 0);
                real_inverse<N>(fa, fb, twY, twX + CLS * 32 + RealRows<N>::SCRATCH * g, j1, g & 1, v);
                float* row = reinterpret_cast<float*>(dst) + (long long)x * DY + Q * j1;
                if (Q == 2 || !p.rows16) {
#pragma unroll
                    for (int j = 0; j < K1; ++j)
#pragma unroll
                        for (int q = 0; q < Q; q += 2) {
                            const float2 s0 = v[q][real_slot<N>(j)], s1 = v[q + 1][real_slot<N>(j)];
                            *reinterpret_cast<float2*>(row + 16 * j + q) = make_float2(s0.x, s1.x);
                            *reinterpret_cast<float2*>(row + DY + 16 * j + q) = make_float2(s0.y, s1.y);
                        }
                } else if constexpr (Q == 4) {
#pragma unroll
                    for (int j = 0; j < K1; ++j) {
                        const int at = real_slot<N>(j);
                        *reinterpret_cast<float4*>(row + 16 * j) = make_float4(v[0][at].x, v[1][at].x, v[2][at].x, v[3][at].x);
                        *reinterpret_cast<float4*>(row + DY + 16 * j) = make_float4(v[0][at].y, v[1][at].y, v[2][at].y, v[3][at].y);
                    }
                }
            } else {
                float2 v[32];
                const float2* line = sY + lr * kModes;
#pragma unroll
                for (int c = 0; c < 16; ++c) folded(line, lr, c, v[2 * c], v[2 * c + 1]);
                fft32<SIGN>(v);
                // Lanes j1 and j1 ^ 1 own samples that alternate in memory: each stores 16 bytes (its own
                // sample and the neighbour's) for every second j2 and they swap the foreign halves with a
                // shuffle, so that a group writes a whole 128-byte line per instruction.
                float2* row = reinterpret_cast<float2*>(dst) + (long long)x * DY + (odd ? RY : 0) + (j1 & ~1);
#pragma unroll
                for (int n2 = 0; n2 < 16; ++n2) {
                    const float2 ev = v[slot32(2 * n2)], od = v[slot32(2 * n2 + 1)];
                    const float2 got = shfl_xor2(odd ? ev : od, 1);
                    *reinterpret_cast<float4*>(row + 2 * RY * n2) =
                        odd ? make_float4(got.x, got.y, od.x, od.y) : make_float4(ev.x, ev.y, got.x, got.y);
                }
            }
        }
        __syncthreads();
    }
}

// The same on the 64-point transform (DX = 64 RX, DY = 64 RY): a thread holds a whole column or 64 samples of a
// row, so half as many lanes read each row's 64 modes from shared memory, at 255 registers and eight warps per SM.
// Two CTAs of 128 threads (CLS = 2 residue classes of 64 rows) share an SM.  The direction is a run-time branch on
// purpose: it keeps the compiler from moving the loads of the modes into the arithmetic, which costs 50 registers
// and spills (246 against 233 us for 4096 images of 128 x 256).
template <int RX, int RY, int CLS, bool CENTERED_X>
__global__ void __launch_bounds__(64 * CLS, 1) ifft2d_pad64_kernel(ImageParams p) {
    constexpr int T = 64 * CLS, ROWS = 64 * CLS, PARTS = RX / CLS, DX = 64 * RX, DY = 64 * RY;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* sY = reinterpret_cast<float2*>(smem_raw);           // [ROWS][64] swizzled
    float2* twY = sY + ROWS * kModes;                            // [RY][64]
    float2* twX = twY + RY * 64;                                 // [CLS][64]
    const int tid = threadIdx.x;
    const int part = PARTS == 1 ? 0 : (int)(blockIdx.x % PARTS);     // the grid is a multiple of PARTS
    fill_inverse_table<RY>(twY, tid, T, make_float2(1.f, 0.f), p.conj_inverse != 0);
    for (int i = tid; i < CLS * 64; i += T) {                    // rows part*CLS .. of fill_inverse_table<RX>
        const int jl = i >> 6, m = i & 63, j1 = part * CLS + jl;
        const int e = CENTERED_X ? (j1 * m - 32 * j1) & (DX - 1) : (j1 * m) & (DX - 1);
        twX[tw_index<CLS>(jl, m)] = cmul(p.gain, unit_root(e, DX, p.conj_inverse ? 1.0f : -1.0f));
    }
    __syncthreads();
    const int ky = tid & 63, jl = tid >> 6;
    const int g = tid / RY, j1 = tid % RY;
    follow_previous_kernel();
    for (long long img = blockIdx.x / PARTS; img < p.nimg; img += gridDim.x / PARTS) {
        if (gridDim.x / PARTS >= p.nimg) admit_next_kernel();
        {
            const float2* src = p.in + img * (long long)(kModes * kModes) + ky;
            float2 v[64];
#pragma unroll
            for (int m = 0; m < 64; ++m) v[m] = load_global(src + m * kModes);
            if (p.conj_inverse) inverse_pad_lane<+1, CLS, CENTERED_X>(v, twX, jl);
            else inverse_pad_lane<-1, CLS>(v, twX, jl);
#pragma unroll
            for (int j2 = 0; j2 < 64; ++j2) {
                const int row = j2 * CLS + jl;
                sY[row * kModes + rtile_chunk(row, ky >> 1) * 2 + (ky & 1)] = v[slot(j2)];
            }
        }
        __syncthreads();
        float2* dst = p.out + (img % p.per_k) * p.stride_b + (img / p.per_k) * p.stride_k + (long long)(part * CLS) * DY;
#pragma unroll 1
        for (int x0 = 0; x0 < ROWS; x0 += T / RY) {
            const int lr = x0 + g;
            const float2* line = sY + lr * kModes;
            float2 v[64];
#pragma unroll
            for (int c = 0; c < 32; ++c) {
                const float4 q = *reinterpret_cast<const float4*>(line + rtile_chunk(lr, c) * 2);
                v[2 * c] = make_float2(q.x, q.y);
                v[2 * c + 1] = make_float2(q.z, q.w);
            }
            if (p.conj_inverse) inverse_pad_lane<+1, RY>(v, twY, j1);
            else inverse_pad_lane<-1, RY>(v, twY, j1);
            store_decimated_paired<RY>(v, dst + (RX * (lr / CLS) + lr % CLS) * DY, j1);
        }
        __syncthreads();
    }
}
#endif

}  // namespace tfno
