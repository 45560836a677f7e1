// Launches of the whole-image transforms (kernels: spectral_image.cuh).
#include "spectral_image.cuh"

namespace tfno {
namespace {

template <int RX, int RY, int C, bool REAL>
int launch_forward(const DeviceInfo& dev, const ImageParams& p, cudaStream_t st) {
    constexpr int THREADS = 64 * RX / C;
    auto kernel = fft2d_trunc_kernel<RX, RY, C, REAL>;
    const size_t smem = unshared_smem(dev, p.nimg * C, fwd_image_smem_bytes<RX, RY, C, REAL>());
    if ((long long)smem > dev.max_smem_optin) return TFNO_ERR_UNSUPPORTED;
    if (record_launch(dev, "fft2d_trunc_kernel<%d,%d,%d>", RX, RY, C)) return TFNO_OK;
    int occ = 0;
    const int rc = prepare_kernel(kernel, smem, dev, &occ, THREADS);
    if (rc != TFNO_OK) return rc;
    // a cluster of CTAs per image, or as many CTAs as are resident together
    long long clusters = p.nimg;
    if (C == 1 && clusters > (long long)dev.sms * occ) clusters = (long long)dev.sms * occ;
    return launch_chained(kernel, dim3((unsigned)(clusters * C)), THREADS, smem, st, clusters == p.nimg && clusters * C <= dev.sms, C, p);
}
// A cluster of CTAs of 64 rows per image, or one CTA per image.  The cluster takes an image at a time, so its launches have no
// last wave to speak of, but the exchange through distributed shared memory costs more per image:
//   - while two such CTAs per SM cover the images: us, cluster / one CTA, 80 images of 128 x 256 11.6 / 11.7, of 256 x 256 16.1 / 18.9,
//     of 256 x 128 15.4 / 16.2, of 128 x 128 11.0 / 10.9; a few images up to twice as fast (16 of 256 x 256 9.2 / 16.7);
//   - beyond one wave of images, where one CTA per image would leave more of its last wave empty than the exchange costs (rows of
//     256 samples 16 %, 20 % for real samples or two images per SM; rows of 128, which shuffle on both sides, 45 %; of 128 x 128 and
//     real ones never).  256 x 256: 152 images 28.4 / 37.0, 200 33.9 / 37.8, 296 46.2 / 41.6, 448 62.3 / 69.5, 512 68.6 / 71.3, 592 77.6 /
//     72.5; real 152 21.1 / 27.7, 448 47.0 / 50.9, 512 52.0 / 51.1.  128 x 256: 320 29.1 / 30.0, 448 35.9 / 37.1, 512 39.6 / 38.5.  256 x 128: 152
//     24.0 / 29.8, 200 28.9 / 30.1, 320 44.0 / 42.7; real 152 21.8 / 21.1.  128 x 128: 320 23.1 / 23.0, 448 29.9 / 29.1.
template <int RX, int RY, bool REAL>
bool image_clusters(const DeviceInfo& dev, long long images) {
    if (images * (RX / 2) <= 2LL * dev.sms) return true;
    constexpr int COST = RY == 8 ? (REAL || RX == 4 ? 120 : 116) : REAL || RX == 4 ? 0 : 145;      // per cent of one CTA's time per image
    const long long wave = dev.sms * (RX == 8 ? 1LL : 2LL);
    return COST && images > wave && images * COST < 100 * ((images + wave - 1) / wave) * wave;
}
template <int RX, int RY, bool REAL>
int launch_forward_split(const DeviceInfo& dev, const ImageParams& p, cudaStream_t st) {
    if (image_clusters<RX, RY, REAL>(dev, p.nimg)) return launch_forward<RX, RY, RX / 2, REAL>(dev, p, st);
    return launch_forward<RX, RY, 1, REAL>(dev, p, st);
}

template <int RX, int RY, int CLS, bool INVERSE, bool REAL>
int launch_inverse(const DeviceInfo& dev, const ImageParams& p, cudaStream_t st) {
    constexpr int PARTS = RX / CLS, THREADS = 64 * CLS;
    auto kernel = ifft2d_pad_kernel<RX, RY, CLS, INVERSE, REAL>;
    const size_t smem = unshared_smem(dev, p.nimg * PARTS, inv_image_smem_bytes<RY, CLS, REAL>());
    if ((long long)smem > dev.max_smem_optin) return TFNO_ERR_UNSUPPORTED;
    if (record_launch(dev, "ifft2d_pad_kernel<%d,%d,%d,%d>", RX, RY, CLS, INVERSE)) return TFNO_OK;
    int occ = 0;
    const int rc = prepare_kernel(kernel, smem, dev, &occ, THREADS);
    if (rc != TFNO_OK) return rc;
    long long images = (long long)dev.sms * occ / PARTS;
    if (images > p.nimg) images = p.nimg;
    return launch_chained(kernel, dim3((unsigned)(images * PARTS)), THREADS, smem, st, images == p.nimg && images * PARTS <= dev.sms, 1, p);
}

template <int RX, bool CENTERED_X>
int launch_inverse64(const DeviceInfo& dev, const ImageParams& p, cudaStream_t st) {        // DX = 64 RX, DY = 256
    constexpr int CLS = 2, PARTS = RX / CLS, THREADS = 64 * CLS;
    auto kernel = ifft2d_pad64_kernel<RX, 4, CLS, CENTERED_X>;
    const size_t smem = unshared_smem(dev, p.nimg * PARTS, inv64_image_smem_bytes<4, CLS>());
    if ((long long)smem > dev.max_smem_optin) return TFNO_ERR_UNSUPPORTED;
    if (record_launch(dev, "ifft2d_pad64_kernel<%d,%d,%d,%d>", RX, 4, CLS, CENTERED_X)) return TFNO_OK;
    int occ = 0;
    const int rc = prepare_kernel(kernel, smem, dev, &occ, THREADS);
    if (rc != TFNO_OK) return rc;
    long long images = (long long)dev.sms * occ / PARTS;
    if (images > p.nimg) images = p.nimg;
    return launch_chained(kernel, dim3((unsigned)(images * PARTS)), THREADS, smem, st, images == p.nimg && images * PARTS <= dev.sms, 1, p);
}

template <int RX, int RY, int CLS>
int launch_image(const DeviceInfo& dev, const ImageParams& p, bool inverse, cudaStream_t st) {
    if (!inverse) return p.real ? launch_forward_split<RX, RY, true>(dev, p, st) : launch_forward_split<RX, RY, false>(dev, p, st);
    if (p.real) return launch_inverse<RX, RY, CLS, true, true>(dev, p, st);
    if constexpr (RY == 8) {
        // More CTAs than the 64-point kernel has resident (two per SM, RX/4 per image): its throughput decides
        // (8192 images of 256 x 256: 880 against 993 us).  Fewer: the smaller parts of the 32-point kernel.
        if (p.nimg * (RX / 4) > 2LL * dev.sms)
            return p.centered_x && p.conj_inverse ? launch_inverse64<RX / 2, true>(dev, p, st) : launch_inverse64<RX / 2, false>(dev, p, st);
    }
    return p.conj_inverse ? launch_inverse<RX, RY, CLS, true, false>(dev, p, st) : launch_inverse<RX, RY, CLS, false, false>(dev, p, st);
}

}  // namespace

bool fft2d_fits(const DeviceInfo& dev) {
    return (long long)fwd_image_smem_bytes<8, 8, 1, false>() <= dev.max_smem_optin;      // the largest of the instances below
}

// Residue classes per inverse CTA: two (128 threads) except at 256 x 256, where four (256 threads, half as many
// reads of the spectrum) take 993 against 1013 us for 8192 images; at 256 x 128 two take 307 against 333 us for 4096,
// and all eight in one CTA of 512 threads take 1173 and 380 us.
int launch_fft2d(const DeviceInfo& dev, int DX, int DY, const ImageParams& params, bool inverse, cudaStream_t st) {
    ImageParams p = params;
    if (p.nimg <= 0) return TFNO_OK;
    const void* full = inverse ? (const void*)p.out : (const void*)p.in;
    if ((reinterpret_cast<uintptr_t>(full) & 15) != 0 || (p.stride_b & 1) != 0 || (p.stride_k & 1) != 0) return TFNO_ERR_UNSUPPORTED;
    if (p.real && inverse && !p.conj_inverse) return TFNO_ERR_UNSUPPORTED;
    p.rows16 = p.real && ((p.stride_b | p.stride_k) & 3) == 0 ? 1 : 0;       // even strides are 16 bytes of complex samples, 8 of real ones
    if (DX == 128 && DY == 128) return launch_image<4, 4, 2>(dev, p, inverse, st);
    if (DX == 128 && DY == 256) return launch_image<4, 8, 2>(dev, p, inverse, st);
    if (DX == 256 && DY == 128) return launch_image<8, 4, 2>(dev, p, inverse, st);
    if (DX == 256 && DY == 256) return launch_image<8, 8, 4>(dev, p, inverse, st);
    return TFNO_ERR_UNSUPPORTED;
}

}  // namespace tfno
