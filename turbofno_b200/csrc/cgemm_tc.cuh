// Channel contraction of compact spectra on the 5th-generation tensor cores:
//
//     C[m + n*M] = alpha * sum_k W[k,n] * A[m + k*M],      m < M = TN * tiles,  n < 64,  K <= 64 (TN = 128) or 96 (TN = 64)
//
// the stand-alone CGEMM of the path (reference: fusion_variants/1D_E_baseline/cgemm.cuh:4-205, a
// SIMT FP32 kernel), used between the two image transforms of the 2-D layer and between the row transforms of wide 1-D
// layers.  The weights sit in tensor memory as the A operand for the whole kernel, a tile of the spectra is the B operand
// S[mode][kk] (K-major, tf32 hi and lo parts), fp32 accuracy from three tf32 products:
//
//   warps 0-7    convert  chunks of 16 channels x TN modes (rows of TN*8 bytes brought by cp.async.bulk): a lane takes four
//                         channels of one mode (twice), splits the values into tf32 hi/lo and stores each part as the 16-byte
//                         line of a core matrix.  TN = 128: all eight warps share a chunk; TN = 64: four warps each take every second one.
//   warps 8-11   results  tcgen05.ld of one accumulator row per thread (rows 2n, 2n + 1 = Re, Im of channel n), Re and Im
//                         meet through a shuffle of adjacent lanes and pass through shared memory, so that a store instruction
//                         writes 256 contiguous bytes of two channels
//   warps 12-13  producers  a ring of 6 stages (96 KB at TN = 128), chunks in turn: a copy costs its warp ~130 cycles
//   warp 14      MMA      D[128 x TN modes] += Wt[128 x 8] * S[8 x TN], three products per k-step
//
// Against the form it replaces (four convert warps with 4-byte stores of one chunk per half-team, results through Re/Im planes of
// 64 KB): 64 channels, 28672 modes 17.2 -> 16.0 us, 65536 25.5 -> 24.2, 524288 133 -> 122 (2D layer of 128 x 64 images 129 -> 117; 82 at copy
// speed).  Bound by the MMA thread: an instruction of this shape takes it 80 cycles (48 a
// tile), a chunk another 450 for its barriers and commit; so 16 channels per chunk and not 8 (144 us).  Tried: stores straight
// from the accumulator rows, 32 bytes of sixteen channels each (202 us), landing buffers in registers (146) and private rings
// of 16-byte asynchronous copies (124).
//
// TN = 128 modes per tile when M is a multiple of 128 and there are enough tiles, else 64: one tcgen05.mma of this shape costs
// about the same for 64 and for 128 columns.
//
// Ring stage s and S buffer b take the chunks g = s, b (mod their count) in turn, and every waiter of their barriers sees
// all phases.  Every wait is bounded (see tc::mbar_wait).
#pragma once
#include "spectral_tc.cuh"

namespace tfno {
namespace tcg {

using namespace tc;

constexpr int kGemmThreads = 480;        // 15 warps
constexpr int kConvWarps = 8;
constexpr int kProducers = 2;
constexpr int kCH = 16;                  // channels per chunk; the last one of a tile may have 8
constexpr int kGemmStages = 6;
constexpr unsigned kGemmIdleNs = 64;
constexpr int kOutStride = 32 * 8 + 32;  // bytes per channel of a result warp's staging (32 modes): the four channels of a quarter-warp cover all banks
constexpr int kOutBytes = 16 * kOutStride;
template <int TN> struct GemmGeom {
    static constexpr int ROW_BYTES = TN * 8;                 // TN modes of one channel
    static constexpr int STAGE_BYTES = kCH * ROW_BYTES;
    static constexpr int S_BUFFERS = 384 / TN;
    static constexpr int PART_BYTES = 2 * kCH * TN * 4;      // hi or lo of one chunk: [Re|Im][four channels][mode] 16-byte lines
    static constexpr int LBO = TN * 16, SBO = 128;           // from four channels to the next four, from eight modes to the next eight
    static constexpr int TEAM_WARPS = TN / 16;               // a lane converts four channels of one mode
    static constexpr int TEAMS = kConvWarps / TEAM_WARPS;    // chunks converted at the same time
};

struct CgemmTcParams {
    long long tiles;                     // M / TN
    int K;
    const float2* a; long long a_stride_k;       // A[m + k * a_stride_k]
    const float2* w; long long w_stride_k, w_stride_n;
    float2* c; long long c_stride_n;             // C[m + n * c_stride_n]
    float2 alpha;
    int conj_w;                          // the weights enter conjugated
    int* status;
};

template <int TN>
__host__ inline size_t cgemm_tc_smem_bytes() {
    using G = GemmGeom<TN>;
    // S buffers, ring, staging of the four result warps, barriers with tmem base and abort flag, slack for the alignment of the base
    return (size_t)G::S_BUFFERS * 2 * G::PART_BYTES + (size_t)kGemmStages * G::STAGE_BYTES + 4 * kOutBytes + 512 + 1024;
}

// ADD: C += alpha A W (the second of two launches over the halves of the channels)
template <int TN, bool ADD>
__global__ void __launch_bounds__(kGemmThreads, 1) cgemm_tc_kernel(CgemmTcParams p) {
    static_assert(TN == 64 || TN == 128, "tile of 64 or 128 modes");
    using G = GemmGeom<TN>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int K = p.K;                            // a multiple of 8
    const int NC = (K + kCH - 1) / kCH;           // chunks per tile
    unsigned char* sS = base;                                       // [buffer][hi | lo]
    unsigned char* ring = sS + G::S_BUFFERS * 2 * G::PART_BYTES;
    unsigned char* ostage = ring + kGemmStages * G::STAGE_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(ostage + 4 * kOutBytes);
    constexpr int B_FULL = 0, B_EMPTY = kGemmStages, B_SFULL = 2 * kGemmStages, B_SEMPTY = B_SFULL + G::S_BUFFERS,
                  B_AFULL = B_SEMPTY + G::S_BUFFERS, B_AEMPTY = B_AFULL + 2, B_DRAIN = B_AEMPTY + 2, B_COUNT = B_DRAIN + 1;
    static_assert(B_COUNT * 8 + 8 <= 512, "room for the barriers");
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + B_COUNT);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const uint32_t bar0 = smem_u32(bars);
    auto bar = [&](int i) { return bar0 + 8u * (uint32_t)i; };

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr int kProducerWarp = 12, kMmaWarp = kProducerWarp + kProducers;

    if (tid == 0) {
        for (int s = 0; s < kGemmStages; ++s) { mbar_init(bar(B_FULL + s), 1); mbar_init(bar(B_EMPTY + s), G::TEAM_WARPS); }
        for (int b = 0; b < G::S_BUFFERS; ++b) { mbar_init(bar(B_SFULL + b), G::TEAM_WARPS); mbar_init(bar(B_SEMPTY + b), 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(bar(B_AFULL + b), 1); mbar_init(bar(B_AEMPTY + b), 4); }
        mbar_init(bar(B_DRAIN), 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const uint32_t TM_WHI = 0, TM_WLO = 2 * K, TM_ACC = 4 * K;      // 4 K + 2 TN <= 512 columns
    follow_previous_kernel();
    admit_next_kernel();

    const long long first = blockIdx.x;
    const int n_it = first < p.tiles ? (int)((p.tiles - first + gridDim.x - 1) / gridDim.x) : 0;

    const uint32_t total = (uint32_t)n_it * (uint32_t)NC;            // chunk g of the CTA is chunk g % NC of its tile g / NC

    if (warp >= kProducerWarp && warp < kMmaWarp) {
        // fill the ring from the start, each producer every second chunk
        bool ok = true;
        int c = warp - kProducerWarp;
        const float2* tile_src = p.a + (long long)(lane & (kCH - 1)) * p.a_stride_k + first * TN;
        uint32_t g = (uint32_t)c;
        for (; g < total && ok; g += kProducers, c += kProducers) {
            while (c >= NC) { c -= NC; tile_src += (long long)gridDim.x * TN; }
            const int s = (int)(g % kGemmStages);
            ok = __all_sync(0xffffffffu, mbar_wait(bar(B_EMPTY + s), ((g / kGemmStages) & 1) ^ 1, abort_flag, p.status, 73, kGemmIdleNs));
            if (!ok) break;
            const int valid = K - c * kCH < kCH ? K - c * kCH : kCH;
            if (lane == 0) mbar_arrive_expect_tx(bar(B_FULL + s), valid * G::ROW_BYTES);
            __syncwarp();
            if (lane < valid)
                bulk_load(smem_u32(ring + s * G::STAGE_BYTES + lane * G::ROW_BYTES), tile_src + (long long)(kCH * c) * p.a_stride_k, G::ROW_BYTES, bar(B_FULL + s));
        }
        if (*abort_flag) {
            // copies already issued still write into this CTA's shared memory: let them land
            for (uint32_t j = g >= kGemmStages ? g - kGemmStages : (uint32_t)(warp - kProducerWarp); j < g; j += kProducers)
                mbar_drain(bar(B_FULL + (int)(j % kGemmStages)), (j / kGemmStages) & 1);
        }
    } else {
        // Weights (times alpha) into tensor memory.  Row i = 2 n + part produces Re or Im of output channel n.  All warps but the
        // producers fetch them as contiguous runs with asynchronous 8-byte copies (one trip to memory) into the S buffers, which
        // nothing uses yet, as [n][K channels + 16 bytes], and warps 0-11 (three per TMEM quarter) convert from there.
        constexpr int kStagers = kGemmThreads - 32 * kProducers;
        static_assert(G::S_BUFFERS * 2 * G::PART_BYTES >= 64 * ((TN == 64 ? 96 : 64) * 8 + 16), "weight staging area");
        auto stagers_sync = [] { asm volatile("bar.sync 1, %0;" ::"n"(kStagers) : "memory"); };
        unsigned char* wst = sS;
        const int wrow = K * 8 + 16;
        const bool k_fast = p.w_stride_k == 1;
        const int stid = warp < kProducerWarp ? tid : tid - 32 * kProducers;
#pragma unroll 1
        for (int idx = stid; idx < 64 * K; idx += kStagers) {
            const int kk = k_fast ? idx % K : idx >> 6, nn = k_fast ? idx / K : idx & 63;
            const float2* src = p.w + (long long)kk * p.w_stride_k + (long long)nn * p.w_stride_n;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(wst + nn * wrow + kk * 8)), "l"(src) : "memory");
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        stagers_sync();
        if (warp < kProducerWarp) {
            const int i = 32 * (warp & 3) + lane, n = i >> 1, im_row = i & 1;
            const uint32_t trow = tmem + ((uint32_t)((warp & 3) * 32) << 16);
            for (int c = warp >> 2; c < K / 8; c += 3) {             // eight channels: columns [Xr | Xi]
#pragma unroll
                for (int part = 0; part < 2; ++part) {
                    uint32_t hi[8], lo[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        float2 w1 = *reinterpret_cast<const float2*>(wst + n * wrow + (8 * c + j) * 8);
                        if (p.conj_w) w1.y = -w1.y;
                        w1 = cmul(w1, p.alpha);
                        // Re row: [ Wr | -Wi ],  Im row: [ Wi | Wr ]  against  S = [ Ar ; Ai ]
                        const float x = im_row ? (part ? w1.x : w1.y) : (part ? -w1.y : w1.x);
                        tf32_parts(x, hi[j], lo[j]);
                    }
                    const uint32_t col = (uint32_t)(16 * c + 8 * part);
                    TFNO_TMEM_ST8(trow + TM_WHI + col, hi);
                    TFNO_TMEM_ST8(trow + TM_WLO + col, lo);
                }
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        }
        tc_fence_before();
        stagers_sync();
        tc_fence_after();
    }

    if (warp >= kConvWarps && warp < kProducerWarp) {
        // ---------------- results: accumulator rows -> C ----------------
        const int q = warp & 3;
        const bool odd = (lane & 1) != 0;
        unsigned char* out = ostage + q * kOutBytes;
        float4* put = reinterpret_cast<float4*>(out + (lane >> 1) * kOutStride + (odd ? 16 : 0));
        const float4* get = reinterpret_cast<const float4*>(out + (lane >> 4) * kOutStride + (lane & 15) * 16);
        // ADD: C of the next 32 modes is on its way while these are staged (a load right ahead of its sum waits for memory
        // eight times in a row, behind the stores: 8192 rows, 128 -> 64 channels 661 us)
        float4 prev[8];
        auto fetch = [&](const float2* from) {
#pragma unroll
            for (int i = 0; i < 8; ++i) prev[i] = *reinterpret_cast<const float4*>(from + (long long)(2 * i) * p.c_stride_n);
        };
        bool ok = true;
        for (int it = 0; it < n_it && ok; ++it) {
            const int buf = it & 1;
            float2* ctile = p.c + (long long)(16 * q + (lane >> 4)) * p.c_stride_n + (first + (long long)it * gridDim.x) * TN + 2 * (lane & 15);
            if (ADD && it == 0) fetch(ctile);
            ok = __all_sync(0xffffffffu, mbar_wait(bar(B_AFULL + buf), (it >> 1) & 1, abort_flag, p.status, 71, kGemmIdleNs));
            if (!ok) break;
            tc_fence_after();
            const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + TM_ACC + TN * buf;
#pragma unroll 1
            for (int c0 = 0; c0 < TN; c0 += 32) {
                uint32_t acc[32];
                TFNO_TMEM_LD16(taddr + c0, acc, 0);
                TFNO_TMEM_LD16(taddr + c0 + 16, acc, 16);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                __syncwarp();                      // the staging buffer has been read
                if (c0 + 32 == TN) {
                    tc_fence_before();
                    if (lane == 0) mbar_arrive(bar(B_AEMPTY + buf));
                }
                // four modes: the even lane (Re) keeps the first two, the odd lane (Im) the other two
#pragma unroll
                for (int m = 0; m < 32; m += 4) {
                    const uint32_t s0 = odd ? acc[m] : acc[m + 2], s1 = odd ? acc[m + 1] : acc[m + 3];
                    const float g0 = __uint_as_float(__shfl_xor_sync(0xffffffffu, s0, 1)), g1 = __uint_as_float(__shfl_xor_sync(0xffffffffu, s1, 1));
                    const float k0 = __uint_as_float(odd ? acc[m + 2] : acc[m]), k1 = __uint_as_float(odd ? acc[m + 3] : acc[m + 1]);
                    put[m / 2] = odd ? make_float4(g0, k0, g1, k1) : make_float4(k0, g0, k1, g1);
                }
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 8; ++i) {                // channels 2 i, 2 i + 1 of the warp
                    float4 o = get[i * (2 * kOutStride / 16)];
                    float4* dst = reinterpret_cast<float4*>(ctile + (long long)(2 * i) * p.c_stride_n + c0);
                    if (ADD) { o.x += prev[i].x; o.y += prev[i].y; o.z += prev[i].z; o.w += prev[i].w; }
                    *dst = o;
                }
                if (ADD && (c0 + 32 < TN || it + 1 < n_it))
                    fetch(c0 + 32 < TN ? ctile + c0 + 32 : ctile + (long long)gridDim.x * TN);
            }
        }
    } else if (warp == kMmaWarp && lane == 0) {
        const uint32_t idesc = make_idesc_tf32(TN);
        const uint64_t desc0 = make_kmajor_desc(smem_u32(sS), G::LBO, G::SBO);
        bool ok = true;
        uint32_t g = 0;
        for (int it = 0; it < n_it && ok; ++it) {
            const int buf = it & 1;
            const uint32_t d_tmem = tmem + TM_ACC + TN * buf;
            for (int c = 0; c < NC; ++c, ++g) {
                const int b = (int)(g % G::S_BUFFERS);
                ok = mbar_wait(bar(B_SFULL + b), (g / G::S_BUFFERS) & 1, abort_flag, p.status, 74);
                if (ok && c == 0) ok = mbar_wait(bar(B_AEMPTY + buf), ((it >> 1) & 1) ^ 1, abort_flag, p.status, 75);
                if (!ok) break;
                tc_fence_after();
                const uint64_t dhi = desc0 + (uint64_t)((b * 2 * G::PART_BYTES) >> 4), dlo = dhi + (uint64_t)(G::PART_BYTES >> 4);
                const uint32_t a_hi = tmem + TM_WHI + 2 * kCH * c, a_lo = tmem + TM_WLO + 2 * kCH * c;
                const int valid = K - c * kCH < kCH ? K - c * kCH : kCH;
#pragma unroll
                for (int h = 0; h < 2; ++h) {                        // eight channels
                    if (8 * h >= valid) break;
#pragma unroll
                    for (int part = 0; part < 2; ++part) {
                        const uint64_t off = (uint64_t)(((part * 4 + h * 2) * G::LBO) >> 4);
                        const uint32_t col = 16 * h + 8 * part;
                        umma_tf32_ts(d_tmem, a_hi + col, dhi + off, idesc, (c | h | part) ? 1u : 0u);
                        umma_tf32_ts(d_tmem, a_lo + col, dhi + off, idesc, 1u);
                        umma_tf32_ts(d_tmem, a_hi + col, dlo + off, idesc, 1u);
                    }
                }
                umma_commit(bar(B_SEMPTY + b));
                if (c == NC - 1) umma_commit(bar(B_AFULL + buf));
            }
        }
        // every MMA issued so far has finished before tensor memory is released
        umma_commit(bar(B_DRAIN));
        mbar_drain(bar(B_DRAIN), 0);
    } else if (warp < kConvWarps) {
        // ---------------- convert: ring rows -> S (tf32 hi / lo, K-major) ----------------
        const int team = warp / G::TEAM_WARPS, tw = warp % G::TEAM_WARPS;
        const int kg = tw & 1, mode = (tw >> 1) * 32 + lane;         // channels 4 kg .. and 8 + 4 kg .. of one mode
        int c = team;
        for (uint32_t g = team; g < total; g += G::TEAMS, c += G::TEAMS) {
            while (c >= NC) c -= NC;
            const bool second = K - c * kCH > 8;
            const int s = (int)(g % kGemmStages), b = (int)(g % G::S_BUFFERS);
            if (!__all_sync(0xffffffffu, mbar_wait(bar(B_FULL + s), (g / kGemmStages) & 1, abort_flag, p.status, 76))) break;
            const float2* src = reinterpret_cast<const float2*>(ring + s * G::STAGE_BYTES) + 4 * kg * TN + mode;
            float2 v[2][4];
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int j = 0; j < 4; ++j) v[h][j] = (h == 0 || second) ? src[(8 * h + j) * TN] : make_float2(0.f, 0.f);
            __threadfence_block();          // the loads have returned before the stage is handed back
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(B_EMPTY + s));
            // this buffer is free once the MMAs of the chunk before in it have completed
            if (!__all_sync(0xffffffffu, mbar_wait(bar(B_SEMPTY + b), ((g / G::S_BUFFERS) & 1) ^ 1, abort_flag, p.status, 77))) break;
            float4* hi = reinterpret_cast<float4*>(sS + b * 2 * G::PART_BYTES) + kg * TN + mode;
            float4* lo = hi + G::PART_BYTES / 16;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (h == 1 && !second) break;
                const float2 (&x)[4] = v[h];
                const float4 rh = make_float4(tf32_hi(x[0].x), tf32_hi(x[1].x), tf32_hi(x[2].x), tf32_hi(x[3].x));
                const float4 ih = make_float4(tf32_hi(x[0].y), tf32_hi(x[1].y), tf32_hi(x[2].y), tf32_hi(x[3].y));
                hi[2 * h * TN] = rh;
                hi[(4 + 2 * h) * TN] = ih;
                lo[2 * h * TN] = make_float4(x[0].x - rh.x, x[1].x - rh.y, x[2].x - rh.z, x[3].x - rh.w);
                lo[(4 + 2 * h) * TN] = make_float4(x[0].y - ih.x, x[1].y - ih.y, x[2].y - ih.z, x[3].y - ih.w);
            }
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(B_SFULL + b));
        }
    }

    // ---------------- teardown ----------------
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

}  // namespace tcg
}  // namespace tfno
