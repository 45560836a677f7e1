// Launches of the row transforms (kernels: spectral_rows.cuh).
#include "spectral_rows.cuh"

namespace tfno {

int launch_fft_rows(const DeviceInfo& dev, int len, const RowsParams& p, cudaStream_t st) {
    const int R = len / 64;
    const long long blocks = (p.nsig + kThreads / (2 * R) - 1) / (kThreads / (2 * R));
    switch (R) {
        case 2: return launch_persistent(dev, fft_rows_trunc_kernel<2>, 0, blocks, p, st, "fft_rows_trunc_kernel<%d>", 2);
        case 4: return launch_persistent(dev, fft_rows_trunc_kernel<4>, 0, blocks, p, st, "fft_rows_trunc_kernel<%d>", 4);
        case 8: return launch_persistent(dev, fft_rows_trunc_kernel<8>, 0, blocks, p, st, "fft_rows_trunc_kernel<%d>", 8);
        case 16: return launch_persistent(dev, fft_rows_trunc_kernel<16>, 0, blocks, p, st, "fft_rows_trunc_kernel<%d>", 16);
    }
    return TFNO_ERR_UNSUPPORTED;
}
int launch_ifft_rows(const DeviceInfo& dev, int len, const RowsParams& p, cudaStream_t st) {
    const int R = len / 64;
    const long long blocks = (p.nsig + kIfftRowsThreads / R - 1) / (kIfftRowsThreads / R);
    switch (R) {
        case 2: return launch_persistent(dev, ifft_rows_pad_kernel<2>, 0, blocks, p, st, "ifft_rows_pad_kernel<%d>", 2, kIfftRowsThreads);
        case 4: return launch_persistent(dev, ifft_rows_pad_kernel<4>, 0, blocks, p, st, "ifft_rows_pad_kernel<%d>", 4, kIfftRowsThreads);
        case 8: return launch_persistent(dev, ifft_rows_pad_kernel<8>, 0, blocks, p, st, "ifft_rows_pad_kernel<%d>", 8, kIfftRowsThreads);
        case 16: return launch_persistent(dev, ifft_rows_pad_kernel<16>, 0, blocks, p, st, "ifft_rows_pad_kernel<%d>", 16, kIfftRowsThreads);
    }
    return TFNO_ERR_UNSUPPORTED;
}

}  // namespace tfno
