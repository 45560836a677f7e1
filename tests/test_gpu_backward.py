"""Gradients of the layers (one library call: tfno_backward) and the real-field layer against autograd in double
precision: one and two dimensions, shared and per-mode weights, batches around the tiles and splits of the sums."""
import pytest

pytestmark = pytest.mark.gpu

# Single-precision transforms and fp32 sums of up to B*64*64 products.  Rounding of the sums grows at most like
# eps * sqrt(terms per accumulator): 6e-8 * sqrt(1e3) = 2e-6; the parity tolerance of the suite is 1e-5.
REL = 4e-6


def _reference(x, w, gy, centered):
    """y, grad_x, grad_w in double precision, through torch.fft and autograd."""
    import torch

    real = not x.is_complex()
    x = x.detach().to(torch.float64 if real else torch.complex128).requires_grad_(True)
    w = w.detach().to(torch.complex128).requires_grad_(True)
    rank = x.dim() - 2
    dims = (-2, -1)[-rank:]
    s = torch.fft.fftn(x, dim=dims)
    if centered:
        s = s.roll(32, dims=-2)
    s = s[(Ellipsis,) + (slice(0, 64),) * rank]
    if real:
        half = torch.ones(64, dtype=torch.float64, device=x.device)
        half[0] = 0.5
        s = 2 * half * s
    m = "xy"[-rank:]
    s = torch.einsum("bk#,kn%->bn#".replace("#", m).replace("%", m if w.dim() > 2 else ""), s, w)
    pad = sum(([0, 0, 0, x.shape[d] - 64] if d == -1 else [0, x.shape[d] - 64] for d in reversed(dims)), [])
    full = torch.view_as_complex(torch.nn.functional.pad(torch.view_as_real(s), pad).contiguous())
    if centered:
        full = full.roll(-32, dims=-2)
    y = torch.fft.ifftn(full, dim=dims)
    if real:
        y = y.real
    grads = torch.autograd.grad(y, (x, w), gy.to(y.dtype))
    return (y,) + grads


def _tensors(B, K, N, signal, per_mode, real, seed=0):
    import torch

    g = torch.Generator(device="cuda").manual_seed(seed)

    def rand(*shape, real=False):
        r = torch.rand(shape + (() if real else (2,)), generator=g, device="cuda") * 2 - 1
        return r if real else torch.view_as_complex(r)

    w = rand(K, N, *((64,) * len(signal) if per_mode else ()))
    return rand(B, K, *signal, real=real), w, rand(B, N, *signal, real=real)


def _run(x, w, gy, centered, **kw):
    import torch

    from turbofno_b200.torch_op import rfft_spectral_conv2d

    x, w = x.detach().requires_grad_(True), w.detach().requires_grad_(True)
    if not x.is_complex():
        y = rfft_spectral_conv2d(x, w)
    elif x.dim() == 3:
        y = torch.ops.turbofno_b200.spectral_conv1d(x, w)
    else:
        y = torch.ops.turbofno_b200.spectral_conv2d(x, w, centered)
    return (y,) + torch.autograd.grad(y, (x, w), gy, **kw)


def _check(got, want):
    for name, a, b in zip(("y", "grad_x", "grad_w"), got, want):
        err = ((a - b).norm() / b.norm()).item()
        assert err <= REL, (name, err)


@pytest.mark.parametrize("B", [1, 7, 33, 300])
@pytest.mark.parametrize("K,N,DY,per_mode", [(64, 64, 128, True), (64, 64, 512, True), (64, 128, 256, False), (128, 64, 1024, False)])
def test_gradients_1d(cuda, B, K, N, DY, per_mode):
    x, w, gy = _tensors(B, K, N, (DY,), per_mode, False, B)
    _check(_run(x, w, gy, False), _reference(x, w, gy, False))


@pytest.mark.parametrize("B", [1, 5])
@pytest.mark.parametrize("DX,DY", [(128, 128), (128, 256), (256, 128), (256, 256)])
@pytest.mark.parametrize("kind", ["shared", "shared_centered", "per_mode", "real"])
def test_gradients_2d(cuda, B, DX, DY, kind):
    centered = kind in ("shared_centered", "real")
    x, w, gy = _tensors(B, 64, 64, (DX, DY), kind in ("per_mode", "real"), kind == "real", B)
    _check(_run(x, w, gy, centered), _reference(x, w, gy, centered))


@pytest.mark.parametrize("DX,DY", [(128, 128), (256, 256)])
def test_real_field_with_few_channels_and_many_images(cuda, DX, DY):
    """K = 8: few images forward (a cluster each); B = 12: 768 images out."""
    from turbofno_b200.torch_op import rfft_spectral_conv2d

    for B in (1, 12):
        x, w, gy = _tensors(B, 8, 64, (DX, DY), True, True, B)
        _check((rfft_spectral_conv2d(x, w),), _reference(x, w, gy, True)[:1])


def test_one_gradient_alone_and_views(cuda):
    """Only x or only w needs a gradient; grad_y expanded, x and w at addresses that are not 16-byte aligned."""
    import torch

    from turbofno_b200.torch_op import rfft_spectral_conv2d

    x, w, gy = _tensors(2, 64, 64, (128, 128), True, True)
    y, gx, gw = _reference(x, w, torch.ones_like(gy), True)
    xo = torch.empty(x.numel() + 1, device=cuda)[1:].view(x.shape)
    xo.copy_(x)
    wo = torch.empty(w.numel() + 1, dtype=w.dtype, device=cuda)[1:].view(w.shape)
    wo.copy_(w)
    assert xo.data_ptr() % 16 and wo.data_ptr() % 16
    rfft_spectral_conv2d(xo.requires_grad_(True), wo).sum().backward()
    rfft_spectral_conv2d(xo.detach(), wo.requires_grad_(True)).sum().backward()
    _check((y, xo.grad, wo.grad), (y, gx, gw))


@pytest.mark.parametrize("real", [False, True])
def test_recorded_backward_gives_the_same_gradients_and_a_graph(cuda, real):
    """create_graph takes the differentiable formulas: same values, and grad_x can be differentiated again."""
    import torch

    x, w, gy = _tensors(2, 64, 64, (128, 128), True, real)
    plain = _run(x, w, gy, True)
    gyr = gy.detach().requires_grad_(True)
    recorded = _run(x, w, gyr, True, create_graph=True)
    _check(recorded, plain)
    # grad_x is linear in grad_y with the layer as its adjoint: d<grad_x, v>/d grad_y is the layer applied to v
    v = torch.ones_like(x)
    again, = torch.autograd.grad(recorded[1], gyr, v)
    _check((again,), _reference(v, w, gy, True)[:1])


def test_backward_operator_has_a_shape_function():
    import torch
    from torch._subclasses.fake_tensor import FakeTensorMode

    import turbofno_b200.torch_op  # noqa: F401

    with FakeTensorMode():
        x, w, gy = (torch.empty(s, dtype=torch.complex64) for s in ((3, 64, 256), (64, 128), (3, 128, 256)))
        gx, gw = torch.ops.turbofno_b200.spectral_conv_backward(gy, x, w, False, True, True)
        assert gx.shape == x.shape and gw.shape == w.shape


def test_calls_that_are_refused(cuda):
    import torch

    import turbofno_b200 as t
    from turbofno_b200.torch_op import rfft_spectral_conv2d

    x, w, gy = _tensors(1, 64, 64, (128, 128), True, True)
    with pytest.raises(ValueError):
        rfft_spectral_conv2d(x, w[..., 0])
    with pytest.raises(TypeError):
        rfft_spectral_conv2d(x, w.real.contiguous())
    plan = t.SpectralConv(2, 1, 128, 64, 64, DX=128, layout="batch_major")           # shared weights: no real form
    with pytest.raises(t.TfnoError):
        plan.exec_real(x, w[..., 0, 0].contiguous())
    plan.close()
    x, w, gy = _tensors(1, 8, 64, (128,), False, False)
    with pytest.raises(t.TfnoError):                                                # grad_x needs K a multiple of 64
        _run(x, w, gy, False)
