// Shared by the translation units of the library: device description, launch set-up cache, and the
// parameters of the image transforms and per-mode contractions with their launch functions.
#pragma once
#include <cuda_runtime.h>
#include <cstdio>
#include <cstring>
#include <mutex>
#include "../../include/turbofno_b200.h"

namespace tfno {

constexpr int kThreads = 256;      // threads per CTA of the row-tile and stand-alone transform kernels
constexpr int kModes = 64;         // retained modes per transformed axis

struct DeviceInfo {
    int device = 0;
    int sms = 0;
    int max_smem_optin = 0;
    bool use_tensor_cores = true;   // tcgen05 fused kernel where its shape limits allow
    int* status = nullptr;          // device word written by kernels whose bounded waits ran out
    // Dry run: when set, every launcher appends the name of the kernel it would launch (separated
    // by ';') and launches nothing.  tfno_plan_kernels reports a plan's kernels this way, from
    // the same dispatch code tfno_exec runs.
    char* record = nullptr;
    size_t record_cap = 0;
};

inline int log2_exact(long long v) {
    int l = 0;
    while ((1LL << l) < v) ++l;
    return ((1LL << l) == v) ? l : -1;
}
inline bool supported_len(int len) { return len == 128 || len == 256 || len == 512 || len == 1024; }

// Appends "name" (printf-style) to the record buffer; true when the caller is a dry run.
inline bool record_launch(const DeviceInfo& dev, const char* fmt, int a = 0, int b = 0, int c = 0, int d = 0) {
    if (!dev.record) return false;
    const size_t used = std::strlen(dev.record);
    if (used + 2 < dev.record_cap) {
        int n = 0;
        if (used) n = std::snprintf(dev.record + used, dev.record_cap - used, ";");
        std::snprintf(dev.record + used + n, dev.record_cap - used - n, fmt, a, b, c, d);
    }
    return true;
}

// Per-kernel launch set-up, done once per (kernel, device, block size, shared-memory size) and
// remembered: the opt-in to more than 48 KB of dynamic shared memory and the resident blocks per
// SM.  A fixed table, no heap: the allocation-free entry point goes through here too.
struct KernelSetupEntry {
    const void* func;
    int device, threads;
    size_t smem;
    int occ;
};
constexpr int kKernelSetupSlots = 512;
inline KernelSetupEntry* kernel_setup_table() {
    static KernelSetupEntry table[kKernelSetupSlots];
    return table;
}
inline std::mutex& kernel_setup_mutex() {
    static std::mutex m;
    return m;
}
inline int kernel_setup_count(int add = 0) {
    static int n = 0;
    n += add;
    return n;
}

inline int prepare_kernel_cached(const void* func, int threads, size_t smem, const DeviceInfo& dev, int* blocks_per_sm) {
    if ((long long)smem > dev.max_smem_optin) return TFNO_ERR_UNSUPPORTED;
    std::lock_guard<std::mutex> lock(kernel_setup_mutex());
    KernelSetupEntry* table = kernel_setup_table();
    const int n = kernel_setup_count();
    size_t opted_in = 48 * 1024;        // largest dynamic shared-memory size this kernel has been opted in to so far
    for (int i = 0; i < n; ++i) {
        if (table[i].func != func || table[i].device != dev.device) continue;
        if (table[i].threads == threads && table[i].smem == smem) {
            *blocks_per_sm = table[i].occ;
            return TFNO_OK;
        }
        if (table[i].smem > opted_in) opted_in = table[i].smem;
    }
    // the attribute is one value per kernel: only ever raise it, or a launch that was set up
    // earlier with a larger size would be refused
    if (smem > opted_in) {
        if (cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
            cudaGetLastError();
            return TFNO_ERR_CUDA;
        }
    }
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, func, threads, smem) != cudaSuccess || occ < 1) {
        cudaGetLastError();
        return TFNO_ERR_CUDA;
    }
    if (n < kKernelSetupSlots) {
        table[n] = KernelSetupEntry{func, dev.device, threads, smem, occ};
        kernel_setup_count(1);
    }
    *blocks_per_sm = occ;
    return TFNO_OK;
}

template <typename Kernel>
inline int prepare_kernel(Kernel kernel, size_t smem, const DeviceInfo& dev, int* blocks_per_sm, int threads = kThreads) {
    return prepare_kernel_cached(reinterpret_cast<const void*>(kernel), threads, smem, dev, blocks_per_sm);
}

inline int launch_status() { return cudaGetLastError() == cudaSuccess ? TFNO_OK : TFNO_ERR_CUDA; }

// ----------------------------------------------------------------------------------------------
// Transforms of rows (spectral_rows.cuh, rows.cu)
// ----------------------------------------------------------------------------------------------
struct RowsParams {
    long long nsig;            // number of signals
    long long per_k;           // signals per channel (rows): signal s -> channel s / per_k, row s % per_k
    const float2* in;
    float2* out;
    long long stride_row, stride_k;   // strides of the full-length side (complex elements)
    float2 gain;
    int conj_inverse;
};
int launch_fft_rows(const DeviceInfo& dev, int len, const RowsParams& p, cudaStream_t st);
int launch_ifft_rows(const DeviceInfo& dev, int len, const RowsParams& p, cudaStream_t st);

// ----------------------------------------------------------------------------------------------
// Whole-image 2-D transforms (spectral_image.cuh, image.cu)
// ----------------------------------------------------------------------------------------------
struct ImageParams {
    long long nimg;
    long long per_k;                   // images per channel: image i -> channel i / per_k, batch i % per_k
    const float2* in;
    float2* out;
    long long stride_b, stride_k;      // strides of the full-size side
    float2 gain;
    int conj_inverse;
    int real;                          // the full-size side holds float samples (strides in samples)
    int rows16;                        // real rows of 128 samples: images start on 16-byte boundaries, else on 8-byte ones (set by the launch)
    int centered_x;                    // kept X modes are -32..31 (row kx + 32 of the 64 x 64 block) instead of 0..63
};
// DX, DY in {128, 256}; full-size side: 16-byte aligned base, even strides
int launch_fft2d(const DeviceInfo& dev, int DX, int DY, const ImageParams& p, bool inverse, cudaStream_t st);
bool fft2d_fits(const DeviceInfo& dev);      // no launch above needs more shared memory than the device gives

// ----------------------------------------------------------------------------------------------
// Per-mode contractions and weight gradients (cgemm_permode.cuh, permode.cu)
// ----------------------------------------------------------------------------------------------
constexpr int kPmModes = 8;            // adjacent modes per CTA: 64 contiguous bytes of every row of P, Q and O

struct PerModeParams {
    int I, J;                          // J a multiple of 64
    long long red, modes;              // terms of the sum; modes: a multiple of 8
    const float2* p; long long p_sr, p_si;                 // P[r*p_sr + i*p_si + m]
    const float2* q; long long q_sr, q_sj, q_sm;           // Q[r*q_sr + j*q_sj + m*q_sm]
    float2* o; long long o_si, o_sj, o_sm;                 // O[i*o_si + j*o_sj + m*o_sm]
    float2* partial;                   // [splits][I][J][modes] (sum over modes: [splits][I][J]) when splits > 1 or the modes are summed
    float2 alpha;
    float2 alpha0;                     // factor of the modes m % 64 == 0 (real fields: the ky = 0 column)
    int splits;                        // r is dealt to this many CTAs in runs of split_len
    long long split_len;
    int q_vec;                         // Q may be copied 16 bytes (two modes) at a time
    int o_vec;                         // O may be written 16 bytes (two modes) at a time
};

// The launches (permode.cu).  `partial` must hold permode_partial_bytes() when that is not zero.
enum PermodeKind { PERMODE_APPLY, PERMODE_APPLY_CONJ, PERMODE_GRAD, PERMODE_GRAD_SHARED };
size_t permode_partial_bytes(const DeviceInfo& dev, const PerModeParams& p, PermodeKind kind);
int launch_permode(const DeviceInfo& dev, PerModeParams p, PermodeKind kind, cudaStream_t st);

#if defined(__CUDACC__)
// Programmatic dependent launch.  A kernel launched `early` may have CTAs resident while the previous kernel of the stream
// is still finishing.  Only a kernel whose threads ALL call follow_previous_kernel() before they touch global memory may be
// launched so; the call returns when the previous kernel has completed and its writes are visible, so whoever waits for a
// kernel of the chain waits for all before it.  (The copies around the library transforms and the self-test of the bounded
// wait do not call it: they are launched in order.)  admit_next_kernel() may be called after that wait only; the next launch,
// if it is an early one, begins once every CTA has called it or ended.
//
// Early: launches of at most one CTA per SM, and the fused kernel, the per-mode contractions and the weight gradients at any
// length, whose operands bypass the L1 cache (training step of 7 x 64 images of 128 x 128 194 against 201 us).  Longer launches
// of the transforms read through that cache and lose more than they gain when they start beside a kernel that has the shared
// memory: an SM that never drains keeps the division of the two.  1D layer of 1024 x 128 signals of 512 samples as three
// kernels: 40 us more with all of them early; 2D layer of 128 x 64 images 2160 against 2040 us.  The contraction of shared weights
// in several waves: 4 us more of 355.  Gains: three kernels of one image 27.7 -> 19.9 us, a row-tile kernel behind another 14.3 ->
// 12.7, training step of 512 x 64 signals of 512 samples 256 -> 246.
// Admitted at any length: by the fused kernel, the contractions and gradients, and the clusters of the forward images; by the other
// transforms and the row-tile kernel in launches of one wave.
//
// Dynamic shared memory for a launch of `ctas`.  A CTA for every SM or fewer: each asks for more than half of an SM's, so that none
// share one; launched early they would be stacked on the first SMs that become free.  2D layers of one batch item, us, each
// launch in order / early and stacked / early and apart: 64 images of 256 x 256 39.0 / 41.0 / 34.9, 64 of 128 x 128 28.8 / 26.2 /
// 22.9, 16 of 256 x 256 32.8 / 32.6 / 25.6; gradients of 64 images of 128 x 128 with per-mode weights 113 / 118 / 104.
inline size_t unshared_smem(const DeviceInfo& dev, long long ctas, size_t smem) {
    return ctas <= dev.sms && (long long)smem <= dev.max_smem_optin / 2 ? dev.max_smem_optin / 2 + 1024 : smem;
}
template <typename... Params>
inline int launch_chained(void (*kernel)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t st, bool early, int cluster, const Params&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = early ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    if (cudaLaunchKernelEx(&cfg, kernel, args...) != cudaSuccess) {
        cudaGetLastError();
        return TFNO_ERR_CUDA;
    }
    return launch_status();
}
__device__ __forceinline__ void follow_previous_kernel() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void admit_next_kernel() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename Params, typename Kernel>
inline int launch_persistent(const DeviceInfo& dev, Kernel kernel, size_t smem, long long work_blocks,
                             const Params& p, cudaStream_t st, const char* name, int R, int threads = kThreads) {
    if (work_blocks <= 0) return TFNO_OK;
    if (record_launch(dev, name, R)) return TFNO_OK;
    int occ = 0;
    int rc = prepare_kernel(kernel, smem, dev, &occ, threads);
    if (rc != TFNO_OK) return rc;
    long long grid = (long long)dev.sms * occ;
    if (grid > work_blocks) grid = work_blocks;
    return launch_chained(kernel, dim3((unsigned)grid), threads, smem, st, grid == work_blocks && grid <= dev.sms, 1, p);
}

// Ask the L2 for `bytes` of contiguous global memory, one 128-byte line per thread and round.
__device__ __forceinline__ void prefetch_l2_block(const void* base, int bytes, int tid, int nthreads) {
    const char* b = static_cast<const char*>(base);
    for (int off = tid * 128; off < bytes; off += nthreads * 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(b + off));
}
#endif

}  // namespace tfno
