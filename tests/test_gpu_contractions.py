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
