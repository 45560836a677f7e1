// Launches of the per-mode contractions and the weight gradients (kernels: cgemm_permode.cuh).
#include "cgemm_permode.cuh"

namespace tfno {
namespace {

bool is_grad(PermodeKind kind) { return kind == PERMODE_GRAD || kind == PERMODE_GRAD_SHARED; }

long long blocks_per_split(const PerModeParams& p, int nt) {
    return (p.modes / kPmModes) * (p.J / kPmCols) * ((p.I + 8LL * nt - 1) / (8 * nt));
}
// splits of about four ring stages of terms (33 terms are split in two)
long long most_splits(const PerModeParams& p, PermodeKind kind) { return kind == PERMODE_GRAD ? (p.red + 4 * kPmTerms - 1) / (4 * kPmTerms) : 1; }

// Eights of rows i per CTA: as few blocks as 32 rows allow (each reads and splits Q again), padded least: 40 rows of 4096 modes
// as two tiles of 24 126 us, 64 as two of 32 172.  A grid that leaves SMs without work takes smaller tiles, whose CTAs
// finish earlier: 64 modes, 16 rows 7.0 us in tiles of 8 against 9.9 in one of 16, 64 rows 8.0 against 19.3 in tiles of 32.
int tile_eights(const DeviceInfo& dev, const PerModeParams& p, PermodeKind kind) {
    const int blocks = (p.I + 31) / 32;
    int nt = ((p.I + blocks - 1) / blocks + 7) / 8;
    while (nt > 1 && blocks_per_split(p, nt - 1) * most_splits(p, kind) <= 2LL * dev.sms) --nt;
    return nt;
}
int grad_splits(const DeviceInfo& dev, const PerModeParams& p, PermodeKind kind) {
    // two CTAs for every SM and no more: a few in a second wave would double the time
    long long blocks, most;
    if (kind == PERMODE_GRAD_SHARED) {
        blocks = (long long)((p.I + kPmSumTile - 1) / kPmSumTile) * (p.J / kPmSumTile);
        most = (p.red + 3 * kPmSumTerms - 1) / (3 * kPmSumTerms);
    } else {
        blocks = blocks_per_split(p, tile_eights(dev, p, kind));
        most = most_splits(p, kind);
    }
    long long splits = 2LL * dev.sms / blocks;
    if (splits > most) splits = most;
    return splits < 1 ? 1 : (int)splits;
}

// How the products are made, by the number of terms of a sum.  The error of a short sum is that of its products, of which two tf32
// parts hold fewer bits than FP32; the error of a long one is that of its additions, of which the tensor cores leave one for
// eight terms.  Gradient of per-mode weights, 64 -> 64 channels, relative error against 64 bits in 1e-7, FP32 / four products / three:
// 1 term 1.39 / 1.48 / 1.74, 8 terms 1.54 / 1.67 / 1.81, 12 1.63 / 1.68 / 1.83, 16 1.70 / 1.69 / 1.84, 20 1.78 / 1.70 / 1.85, 24
// 1.85 / 1.71 / 1.85, 32 1.98 / - / 1.86, 1024 2.97 / - / 2.05 (1.33 of it is the transforms').  Gradients of a layer of real
// 128 x 128 images, us, as chosen / with three products always: 1 item 94.5 / 100.4, 4 items 122 / 119, 7 155 / 145, 16 220 / 216, 20 272 / 259.
// Gradient of shared weights, blocks of eight modes: 8 blocks 1.62 / 1.78 / 1.92, 16 1.77 / 1.79 / 1.93, 32 2.04 / 1.85 / 1.97, 8192
// 3.44 / - / 2.39; four products take 2 us more of 32.
constexpr long long kPmFmaTerms = 15, kPmFullTerms = 23, kPmSumFullBlocks = 16;
template <int NT, bool CONJ_Q, bool CONJ_O>
int launch_inst(const DeviceInfo& dev, const PerModeParams& p, cudaStream_t st) {
    auto kernel = p.red <= kPmFmaTerms    ? cgemm_permode_kernel<NT, CONJ_Q, CONJ_O, PM_FMA>
                  : p.red <= kPmFullTerms ? cgemm_permode_kernel<NT, CONJ_Q, CONJ_O, PM_FULL>
                                          : cgemm_permode_kernel<NT, CONJ_Q, CONJ_O, PM_SPLIT>;
    constexpr size_t smem = pm_smem_bytes<NT>();
    int occ = 0;
    const int rc = prepare_kernel(kernel, smem, dev, &occ, kPmThreads);
    if (rc != TFNO_OK) return rc;
    const long long grid = blocks_per_split(p, NT) * p.splits;
    if (grid > 0x7fffffffLL) return TFNO_ERR_UNSUPPORTED;
    return launch_chained(kernel, dim3((unsigned)grid), kPmThreads, smem, st, true, 1, p);
}
template <bool CONJ_Q, bool CONJ_O>
int launch_rows(const DeviceInfo& dev, const PerModeParams& p, PermodeKind kind, cudaStream_t st) {
    switch (tile_eights(dev, p, kind)) {
        case 1: return launch_inst<1, CONJ_Q, CONJ_O>(dev, p, st);
        case 2: return launch_inst<2, CONJ_Q, CONJ_O>(dev, p, st);
        case 3: return launch_inst<3, CONJ_Q, CONJ_O>(dev, p, st);
        default: return launch_inst<4, CONJ_Q, CONJ_O>(dev, p, st);
    }
}

int launch_modesum(const DeviceInfo& dev, const PerModeParams& p, cudaStream_t st) {
    int occ = 0;
    auto kernel = p.red <= kPmSumFullBlocks ? cgemm_modesum_kernel<true> : cgemm_modesum_kernel<false>;
    const int rc = prepare_kernel(kernel, kPmSumSmemBytes, dev, &occ, kPmThreads);
    if (rc != TFNO_OK) return rc;
    const unsigned grid = (unsigned)((p.I + kPmSumTile - 1) / kPmSumTile) * (unsigned)(p.J / kPmSumTile) * (unsigned)p.splits;
    return launch_chained(kernel, dim3(grid), kPmThreads, kPmSumSmemBytes, st, true, 1, p);
}

}  // namespace

size_t permode_partial_bytes(const DeviceInfo& dev, const PerModeParams& p, PermodeKind kind) {
    if (!is_grad(kind)) return 0;
    const int splits = grad_splits(dev, p, kind);
    if (kind == PERMODE_GRAD && splits == 1) return 0;
    return sizeof(float2) * (size_t)splits * p.I * p.J * (kind == PERMODE_GRAD_SHARED ? 1 : (size_t)p.modes);
}

int launch_permode(const DeviceInfo& dev, PerModeParams p, PermodeKind kind, cudaStream_t st) {
    if (p.I <= 0 || p.red <= 0) return TFNO_OK;
    if (p.J <= 0 || p.J % 64 != 0 || p.modes % kPmModes != 0) return TFNO_ERR_UNSUPPORTED;
    if (record_launch(dev, "cgemm_permode_kernel")) return TFNO_OK;
    p.q_vec = (p.q_sm == 1 && ((p.q_sr | p.q_sj) & 1) == 0 && (reinterpret_cast<uintptr_t>(p.q) & 15) == 0) ? 1 : 0;
    p.o_vec = (p.o_sm == 1 && ((p.o_si | p.o_sj) & 1) == 0 && (reinterpret_cast<uintptr_t>(p.o) & 15) == 0) ? 1 : 0;
    p.splits = is_grad(kind) ? grad_splits(dev, p, kind) : 1;
    const int unit = kind == PERMODE_GRAD_SHARED ? kPmSumTerms : kPmTerms;
    p.split_len = ((p.red + p.splits - 1) / p.splits + unit - 1) / unit * unit;
    int rc = TFNO_ERR_UNSUPPORTED;
    switch (kind) {
        case PERMODE_APPLY: return launch_rows<false, false>(dev, p, kind, st);
        case PERMODE_APPLY_CONJ: return launch_rows<true, false>(dev, p, kind, st);
        case PERMODE_GRAD: rc = launch_rows<true, true>(dev, p, kind, st); break;
        case PERMODE_GRAD_SHARED: rc = launch_modesum(dev, p, st); break;
    }
    if (rc != TFNO_OK || (kind == PERMODE_GRAD && p.splits == 1)) return rc;
    if (kind == PERMODE_GRAD_SHARED)
        return launch_chained(modesum_reduce_kernel, dim3((unsigned)((p.I * p.J + 31) / 32)), 32 * kPmSumReducers, 0, st, true, 1, p);
    const long long sums = (long long)p.I * p.J * p.modes;
    long long grid = (sums + 255) / 256;
    if (grid > 8LL * dev.sms) grid = 8LL * dev.sms;
    return launch_chained(permode_reduce_kernel, dim3((unsigned)grid), 256, 0, st, true, 1, p);
}

}  // namespace tfno
