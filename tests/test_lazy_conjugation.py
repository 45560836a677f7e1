"""x.conj() is a flag on the memory of x: a tensor that carries it is contiguous, and its address leads to the values
without the conjugation.  Every entry point has to compute with the values, or refuse to write through the flag."""
import ctypes

import numpy as np
import pytest

# single-precision transforms and fp32 sums of up to B*64*64 products, as in the gradient tests; the suite's parity
# tolerance is 1e-5
REL = 4e-6


class _HostLibrary:
    """Row and column transforms of the C interface on host memory: what a kernel sees at the address it is given."""

    def tfno_fft_stride_DY(self, h, log2_len, src, dst, total, stream):
        n = 1 << log2_len
        x = np.ctypeslib.as_array(ctypes.cast(src, ctypes.POINTER(ctypes.c_float)), (total, n, 2)).view(np.complex64)[..., 0]
        out = np.ctypeslib.as_array(ctypes.cast(dst, ctypes.POINTER(ctypes.c_float)), (total, 64, 2)).view(np.complex64)[..., 0]
        out[:] = np.fft.fft(x)[:, :64]
        return 0

    def tfno_fft_stride(self, h, log2_len, src, dst, DY, columns, stream):
        n, images = 1 << log2_len, columns // DY
        x = np.ctypeslib.as_array(ctypes.cast(src, ctypes.POINTER(ctypes.c_float)), (images, n, DY, 2)).view(np.complex64)[..., 0]
        out = np.ctypeslib.as_array(ctypes.cast(dst, ctypes.POINTER(ctypes.c_float)), (images, 64, DY, 2)).view(np.complex64)[..., 0]
        out[:] = np.fft.fft(x, axis=1)[:, :64]
        return 0


@pytest.fixture
def host_library(monkeypatch):
    from types import SimpleNamespace

    from turbofno_b200 import api

    monkeypatch.setattr(api.Handle, "get", classmethod(lambda cls, device=None: SimpleNamespace(lib=_HostLibrary(), _h=None)))
    monkeypatch.setattr(api, "_stream_ptr", lambda stream=None, device=None: None)


def _complex(*shape):
    import torch

    g = torch.Generator().manual_seed(1)
    return torch.view_as_complex(torch.rand(shape + (2,), generator=g) * 2 - 1)


@pytest.mark.parametrize("lazy", [False, True])
def test_spectra_of_the_recorded_formulas(host_library, lazy):
    """The weight gradient of a recorded backward pass is made of these; saved x and grad_y may carry the flag."""
    import torch

    from turbofno_b200 import torch_op

    x, x2 = _complex(2, 3, 128), _complex(1, 2, 128, 256)
    if lazy:
        x, x2 = x.conj(), x2.conj()
        assert x.is_conj() and x.contiguous().is_conj()
    s = torch_op._truncated_spectrum(x)
    assert (s - torch.fft.fft(x)[..., :64]).abs().max() <= 1e-4
    s2 = torch_op._truncated_spectrum2d(x2)
    assert (s2 - torch.fft.fft2(x2)[..., :64, :64]).abs().max() <= 1e-3


def test_an_output_with_the_flag_is_refused(host_library):
    import torch

    from turbofno_b200 import api

    with pytest.raises(TypeError):
        api.fft_stride_DY(_complex(2, 128), torch.empty((2, 64), dtype=torch.complex64).conj(), 2, 128)


@pytest.mark.gpu
@pytest.mark.parametrize("create_graph", [False, True])
@pytest.mark.parametrize("N", [64, 256])                      # 256: beyond the channel counts of the one-call backward
@pytest.mark.parametrize("signal", [(256,), (128, 128)])
def test_gradients_of_a_loss_on_the_conjugate(cuda, signal, N, create_graph):
    import torch

    from test_gpu_backward import _reference, _tensors

    import turbofno_b200.torch_op  # noqa: F401

    x, w, c = _tensors(2, 64, N, signal, False, False)
    xc = x.conj().detach().requires_grad_(True)                # the saved input carries the flag too
    w = w.detach().requires_grad_(True)
    op = torch.ops.turbofno_b200.spectral_conv1d if len(signal) == 1 else torch.ops.turbofno_b200.spectral_conv2d
    y = op(xc, w)
    seen = []
    y.register_hook(lambda g: seen.append(g.is_conj()))
    loss = (y.conj() * c).sum().real
    gx, gw = torch.autograd.grad(loss, (xc, w), create_graph=create_graph)
    assert seen == [True]                                     # autograd hands on a lazy conjugate here
    ref = _reference(x.conj().resolve_conj(), w.detach(), c, False)
    for name, a, b in zip(("y", "grad_x", "grad_w"), (y, gx, gw), ref):
        assert ((a - b).norm() / b.norm()).item() <= REL, name


@pytest.mark.gpu
def test_plans_compute_with_the_values(cuda):
    import torch

    import turbofno_b200 as t
    from test_gpu_backward import _reference, _tensors

    x, w, gy = _tensors(3, 64, 64, (256,), False, False)
    y, gx, gw = _reference(x.conj().resolve_conj(), w.conj().resolve_conj(), gy.conj().resolve_conj(), False)
    plan = t.SpectralConv(1, 3, 256, 64, 64, layout="batch_major")
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    for stream in (None, side):
        got = [plan(x.conj(), w.conj(), stream=stream), torch.empty_like(x), torch.empty_like(w)]
        plan.backward(x.conj(), w.conj(), gy.conj(), got[1], got[2], stream=stream)
        torch.cuda.synchronize()
        for a, b in zip(got, (y, gx, gw)):
            assert ((a - b).norm() / b.norm()).item() <= REL
    with pytest.raises(TypeError):
        plan(x, w, y=torch.empty(plan.out_shape(), dtype=torch.complex64, device=cuda).conj())
    with pytest.raises(TypeError):
        plan.backward(x, w, gy, torch.empty_like(x).conj(), None)
    plan.close()
    plan = t.SpectralConv(1, 3, 256, 64, 64)                   # reference layout, host buffers
    xh, wh = x.transpose(0, 1).contiguous().cpu(), w.T.contiguous().cpu()
    yh = plan.exec_host(xh.conj(), wh.conj(), torch.empty(plan.out_shape(), dtype=torch.complex64))
    assert ((yh.transpose(0, 1).to(cuda) - y).norm() / y.norm()).item() <= REL
    plan.close()
    x, w, gy = _tensors(1, 8, 64, (128, 128), True, True)
    plan = t.SpectralConv(2, 1, 128, 8, 64, DX=128, layout="batch_major", per_mode_weights=True, x_modes_centered=True)
    y, = _reference(x, w.conj().resolve_conj(), gy, True)[:1]
    assert ((plan.exec_real(x, w.conj()) - y).norm() / y.norm()).item() <= REL
    plan.close()
