"""Channel contractions at the edges of their tiles: gradients of per-mode and shared weights whose channel counts are no multiple of
a tile, batches around a ring stage (eight terms, or four blocks of eight modes) and around a split of the sum, against torch in
double precision."""
import pytest

pytestmark = pytest.mark.gpu

# Transforms as in the other GPU tests (eps * log2(DY) ~ 5e-7).  A product of two split values is off by at most
# 3 * 2^-22 = 7e-7 of its size (the dropped lo*lo and the last bit of each lo), independently per product, so their sum
# is off by less than that relative to its norm; the sums of partial results add eps * sqrt(steps) < 1e-6.
REL = 2.5e-6


def _field(g, *shape):
    import torch

    return torch.view_as_complex(torch.rand(shape + (2,), generator=g, device="cuda") * 2 - 1)


@pytest.mark.parametrize("B", [1, 7, 8, 9, 31, 33, 65, 300])
@pytest.mark.parametrize("K,N,per_mode", [(8, 64, True), (72, 64, True), (24, 128, False), (72, 64, False), (136, 192, False)])
def test_weight_gradients_at_tile_edges(cuda, B, K, N, per_mode):
    import torch
    import turbofno_b200 as t

    DY = 128
    g = torch.Generator(device="cuda").manual_seed(B)
    x, gy = _field(g, B, K, DY), _field(g, B, N, DY)
    w = _field(g, K, N, 64) if per_mode else _field(g, K, N)
    plan = t.SpectralConv(1, B, DY, K, N, layout="batch_major", per_mode_weights=per_mode)
    gw = torch.full_like(w, float("nan"))
    plan.backward(x, w, gy, None, gw)
    X, G = (torch.fft.fft(v.to(torch.complex128))[..., :64] for v in (x, gy))
    want = torch.einsum("bkm,bnm->knm" if per_mode else "bkm,bnm->kn", X.conj(), G) / DY
    assert ((gw - want).norm() / want.norm()).item() <= REL
    plan.close()


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_values_that_are_not_finite_stay_in_their_mode_and_output(cuda, value):
    """A weight that is no number spoils its own mode of its own output channel and nothing else."""
    import torch
    import turbofno_b200 as t

    B, K, N, DY = 9, 16, 64, 128
    g = torch.Generator(device="cuda").manual_seed(1)
    x, w = _field(g, B, K, DY), _field(g, K, N, 64)
    plan = t.SpectralConv(1, B, DY, K, N, layout="batch_major", per_mode_weights=True)
    clean = plan(x, w)
    w[3, 5, 17] = value
    y = plan(x, w)
    assert not torch.isfinite(torch.view_as_real(y[:, 5])).any()
    keep = [n for n in range(N) if n != 5]
    assert torch.equal(y[:, keep], clean[:, keep])
    plan.close()


def _not_a_number(kind):
    """On the GPU: a NaN from the host has the payload 0x400000, one that arithmetic made there all bits."""
    import torch

    inf = torch.full((), float("inf"), device="cuda")
    return {"host": torch.full((), float("nan"), device="cuda"), "arithmetic": inf * 0, "negative": -(inf * 0), "inf": inf}[kind]


@pytest.mark.parametrize("kind", ["host", "arithmetic", "negative", "inf"])
@pytest.mark.parametrize("part", [0, 1])
@pytest.mark.parametrize("path", ["fused", "wide", "2d", "grad_x"])
def test_shared_weights_that_are_not_finite_spoil_their_output(cuda, path, part, kind):
    """A shared weight that is no number must not pass for zero on the tensor cores."""
    import torch
    import turbofno_b200 as t

    rank, B, K, N, DY = {"fused": (1, 300, 64, 64, 256), "wide": (1, 300, 64, 128, 512), "2d": (2, 2, 32, 64, 128), "grad_x": (2, 2, 64, 64, 128)}[path]
    sig = (DY,) * rank
    plan = t.SpectralConv(rank, B, DY, K, N, layout="batch_major")
    kernel = "spectral_tc_kernel" if path == "fused" else "cgemm_tc_kernel"
    assert any(k.startswith(kernel) for k in plan.kernels())
    g = torch.Generator(device="cuda").manual_seed(2)
    x, w = _field(g, B, K, *sig), _field(g, K, N)
    if path == "grad_x":
        gy, out, own = _field(g, B, N, *sig), 3, K

        def call():
            gx = torch.empty_like(x)
            plan.backward(x, w, gy, gx, None)
            return gx
    else:
        out, own = 5, N

        def call():
            return plan(x, w)
    clean = call()
    torch.view_as_real(w)[3, 5, part] = _not_a_number(kind)
    y = call()
    assert not torch.isfinite(torch.view_as_real(y[:, out])).any()
    keep = [n for n in range(own) if n != out]
    assert torch.equal(y[:, keep], clean[:, keep])
    plan.close()


@pytest.mark.parametrize("rows", [296, 297, 298, 592, 600])      # tiles of 128 modes (of 64: 297) one, two and a few more than two per SM
@pytest.mark.parametrize("K,N", [(104, 64), (128, 128)])
def test_contraction_in_two_launches_of_which_the_second_adds(cuda, rows, K, N):
    import torch
    import turbofno_b200 as t

    M = 64 * rows
    g = torch.Generator(device="cuda").manual_seed(rows)
    A, w = _field(g, K, M), _field(g, N, K)
    C = torch.full((N, M), float("nan"), dtype=torch.complex64, device=cuda)
    t.api.cgemm(M, N, K, A, w, C)
    want = w.to(torch.complex128) @ A.to(torch.complex128)
    assert ((C - want).norm() / want.norm()).item() <= REL


@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_per_mode_contractions_of_the_largest_floats(cuda, sign):
    """FLT_MAX as a weight, or in the spectrum of a gradient: finite results where the products are."""
    import torch
    import turbofno_b200 as t

    B, K, N, DY = 9, 64, 64, 128
    top = sign * torch.finfo(torch.float32).max
    g = torch.Generator(device="cuda").manual_seed(4)
    small = lambda *s: _field(g, *s) * 2.0 ** -9
    rel = lambda got, want: ((got.to(torch.complex128) - want).abs().max() / want.abs().max()).item()
    spectrum = lambda v: torch.fft.fft(v.to(torch.complex128))[..., :64]
    pad = lambda s: torch.fft.ifft(torch.cat([s, s.new_zeros(*s.shape[:2], DY - 64)], -1))
    x, gy, w = small(B, K, DY), small(B, N, DY), _field(g, K, N, 64)
    w[3, 5, 17] = complex(top, -top)
    plan = t.SpectralConv(1, B, DY, K, N, layout="batch_major", per_mode_weights=True)
    w2 = w.to(torch.complex128)
    # one channel in, one mode: each product is within 4 roundings of 2^-24 and two dropped parts of 2^-22, the transforms as above
    assert rel(plan(x, w)[:, 5], pad(torch.einsum("bkm,knm->bnm", spectrum(x), w2))[:, 5]) <= REL
    # a pulse has FLT_MAX in every mode
    x[2, 7] = 0
    x[2, 7, 0] = top
    gx, gw = torch.empty_like(x), torch.empty_like(w)
    plan.backward(x, w, gy, gx, gw)
    assert rel(gx[:, 3], pad(torch.einsum("bnm,knm->bkm", spectrum(gy), w2.conj()))[:, 3]) <= REL
    assert rel(gw[7], torch.einsum("bkm,bnm->knm", spectrum(x).conj(), spectrum(gy))[7] / DY) <= REL
    plan.close()
    shared = t.SpectralConv(1, B, DY, K, N, layout="batch_major")
    gw = torch.empty(K, N, dtype=torch.complex64, device=cuda)
    shared.backward(x, _field(g, K, N), gy, None, gw)
    assert rel(gw[7], torch.einsum("bkm,bnm->kn", spectrum(x).conj(), spectrum(gy))[7] / DY) <= REL
    shared.close()


@pytest.mark.parametrize("B", [1, 2, 4, 15, 16, 20, 23, 24])
@pytest.mark.parametrize("K", [64, 8])
def test_short_sums_are_as_exact_as_fp32(cuda, B, K):
    """Gradient of per-mode weights against the exact products of the spectra the library itself makes, so that the error is
    that of the contraction.  An FP32 chain of 2 B multiply-adds rounds at the sizes of its partial sums: in the norm
    sqrt(B) times the rms of a rounding, 2.5e-8, and one more at the front.  Two tf32 parts alone make 1.1e-7 of one term."""
    import torch
    import turbofno_b200 as t

    N, DY = 64, 256
    g = torch.Generator(device="cuda").manual_seed(6)
    x, gy, w = _field(g, B, K, DY), _field(g, B, N, DY), _field(g, K, N, 64)
    plan = t.SpectralConv(1, B, DY, K, N, layout="batch_major", per_mode_weights=True)
    gw = torch.empty_like(w)
    plan.backward(x, w, gy, None, gw)
    plan.close()
    X, G = (t.api.fft_stride_DY(v, torch.empty(v.shape[:2] + (64,), dtype=v.dtype, device=cuda), v.shape[0] * v.shape[1], DY).to(torch.complex128) for v in (x, gy))
    want = torch.einsum("bkm,bnm->knm", X.conj(), G) / DY
    assert ((gw.to(torch.complex128) - want).norm() / want.norm()).item() <= 2.5e-8 * (B + 1) ** 0.5 * 1.15
