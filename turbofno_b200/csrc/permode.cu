// Launches of the per-mode contractions and the weight gradients (kernels: cgemm_permode.cuh).
#include "cgemm_permode.cuh"

namespace tfno {
namespace {

// dst[k*N + n] = conj(w[k, n])
__global__ void __launch_bounds__(256) conjugate_kernel(const float2* __restrict__ w, long long sk, long long sn, int K, int N, float2* __restrict__ dst) {
    for (int e = blockIdx.x * 256 + threadIdx.x; e < K * N; e += gridDim.x * 256) {
        const float2 v = w[(e / N) * sk + (e % N) * sn];
        dst[e] = make_float2(v.x, -v.y);
    }
}

// rows i per CTA: the tile that pads the rows least, the larger one of two equals.  At 4096 modes (64 -> 64 and 32 -> 128
// channels, 1 to 48 rows, every tile forced in turn) that is the fastest one up to 36 rows: 1 row 33 us (tile of 8: 42), 8 rows 45
// (4: 54, 12: 54), 12 rows 56 (8: 75, 16: 71), 16 rows 73 (8: 76, 12: 94), 20 rows 94 with 12 (8: 114, 16: 132), 32 rows 125 with 16
// (12: 144); 48 rows 192 with 16 against 184 with 12.  With the 64 modes of a 1D layer and so few rows the grid is a handful of CTAs
// and the smallest tile is the fastest (16 rows: 10.8 us with 4, 20.6 with 16); the rule does not know that.
int tile_rows(int I) {
    int best = 16;
    long long padded = (I + 15LL) / 16 * 16;
    for (int rows = 12; rows >= 4; rows -= 4) {
        const long long n = (I + rows - 1LL) / rows * rows;
        // several blocks of 4 or 8 rows would read Q again, for which the tile is too small
        if (n < padded && (rows == 12 || I <= rows)) { padded = n; best = rows; }
    }
    return best;
}

bool is_grad(PermodeKind kind) { return kind == PERMODE_GRAD || kind == PERMODE_GRAD_SHARED; }

long long blocks_per_split(const PerModeParams& p, int rows) {
    return (p.modes / kPmModes) * (p.J / kPmCols) * ((p.I + rows - 1LL) / rows);
}
int grad_splits(const DeviceInfo& dev, const PerModeParams& p) {
    // two CTAs for every SM, at least eight ring slabs each
    const long long blocks = blocks_per_split(p, tile_rows(p.I));
    long long splits = (2LL * dev.sms + blocks - 1) / blocks;
    const long long most = (p.red + 8 * kPmSlab - 1) / (8 * kPmSlab);
    if (splits > most) splits = most;
    return splits < 1 ? 1 : (int)splits;
}

template <int TI, bool CONJ_Q, bool CONJ_O, bool SUM_MODES>
int launch_inst(const DeviceInfo& dev, const PerModeParams& p, cudaStream_t st) {
    auto kernel = cgemm_permode_kernel<TI, CONJ_Q, CONJ_O, SUM_MODES>;
    constexpr size_t smem = pm_smem_bytes<TI>();
    int occ = 0;
    const int rc = prepare_kernel(kernel, smem, dev, &occ, kPmThreads);
    if (rc != TFNO_OK) return rc;
    const long long grid = blocks_per_split(p, 4 * TI) * p.splits;
    if (grid > 0x7fffffffLL) return TFNO_ERR_UNSUPPORTED;
    kernel<<<(unsigned)grid, kPmThreads, smem, st>>>(p);
    return launch_status();
}
template <bool CONJ_Q, bool CONJ_O, bool SUM_MODES>
int launch_rows(const DeviceInfo& dev, const PerModeParams& p, cudaStream_t st) {
    switch (tile_rows(p.I)) {
        case 4: return launch_inst<1, CONJ_Q, CONJ_O, SUM_MODES>(dev, p, st);
        case 8: return launch_inst<2, CONJ_Q, CONJ_O, SUM_MODES>(dev, p, st);
        case 12: return launch_inst<3, CONJ_Q, CONJ_O, SUM_MODES>(dev, p, st);
        default: return launch_inst<4, CONJ_Q, CONJ_O, SUM_MODES>(dev, p, st);
    }
}

}  // namespace

size_t permode_partial_bytes(const DeviceInfo& dev, const PerModeParams& p, PermodeKind kind) {
    if (!is_grad(kind)) return 0;
    const int splits = grad_splits(dev, p);
    if (kind == PERMODE_GRAD && splits == 1) return 0;
    return sizeof(float2) * (size_t)splits * p.I * p.J * (kind == PERMODE_GRAD_SHARED ? 1 : (size_t)p.modes);
}

int launch_permode(const DeviceInfo& dev, PerModeParams p, PermodeKind kind, cudaStream_t st) {
    if (p.I <= 0 || p.red <= 0) return TFNO_OK;
    if (p.J <= 0 || p.J % kPmCols != 0 || p.modes % kPmModes != 0) return TFNO_ERR_UNSUPPORTED;
    if (record_launch(dev, "cgemm_permode_kernel")) return TFNO_OK;
    p.q_vec = (p.q_sm == 1 && ((p.q_sr | p.q_sj) & 1) == 0 && (reinterpret_cast<uintptr_t>(p.q) & 15) == 0) ? 1 : 0;
    p.splits = is_grad(kind) ? grad_splits(dev, p) : 1;
    p.split_len = ((p.red + p.splits - 1) / p.splits + kPmSlab - 1) / kPmSlab * kPmSlab;
    int rc = TFNO_ERR_UNSUPPORTED;
    switch (kind) {
        case PERMODE_APPLY: return launch_rows<false, false, false>(dev, p, st);
        case PERMODE_APPLY_CONJ: return launch_rows<true, false, false>(dev, p, st);
        case PERMODE_GRAD: rc = launch_rows<true, true, false>(dev, p, st); break;
        case PERMODE_GRAD_SHARED: rc = launch_rows<true, true, true>(dev, p, st); break;
    }
    if (rc != TFNO_OK || (kind == PERMODE_GRAD && p.splits == 1)) return rc;
    const long long sums = (long long)p.I * p.J * (kind == PERMODE_GRAD ? p.modes : 1);
    long long grid = (sums + 255) / 256;
    if (grid > 8LL * dev.sms) grid = 8LL * dev.sms;
    if (kind == PERMODE_GRAD) permode_reduce_kernel<false><<<(unsigned)grid, 256, 0, st>>>(p);
    else permode_reduce_kernel<true><<<(unsigned)grid, 256, 0, st>>>(p);
    return launch_status();
}

int launch_conjugate(const DeviceInfo& dev, const float2* w, long long sk, long long sn, int K, int N, float2* dst, cudaStream_t st) {
    conjugate_kernel<<<(unsigned)((K * N + 255) / 256), 256, 0, st>>>(w, sk, sn, K, N, dst);
    return launch_status();
}

}  // namespace tfno
