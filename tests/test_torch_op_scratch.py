"""Scratch of the torch operators: a plan is shared by all callers of its shape, so every call needs scratch of its own."""
import pytest


class _RecordingPlan:
    """Stands in for SpectralConv: keeps what the operator passes."""

    def __init__(self, nbytes):
        from turbofno_b200.api import SpectralConv

        self.workspace_bytes, self._optional_ws, self.calls = nbytes, False, []
        self._scratch = SpectralConv._scratch
        self.call_scratch = lambda device, stream=None: SpectralConv.call_scratch(self, device, stream)

    def _launch(self, x, w, y, workspace, stream=None):
        self.calls.append((y, workspace))
        return y


@pytest.mark.parametrize("kernel,x_shape,w_shape", [("_conv1d_cuda", (2, 8, 128), (8, 64, 64)), ("_conv2d_cuda", (2, 8, 128, 128), (8, 64))])
def test_every_operator_call_brings_its_own_scratch(monkeypatch, kernel, x_shape, w_shape):
    import torch

    from turbofno_b200 import torch_op

    plan = _RecordingPlan(4096)
    monkeypatch.setattr(torch_op, "_plan", lambda *a, **k: plan)
    x, w = torch.zeros(x_shape, dtype=torch.complex64), torch.zeros(w_shape, dtype=torch.complex64)
    for _ in range(2):
        getattr(torch_op, kernel)(x, w)
    spaces = [ws for _, ws in plan.calls]
    assert all(ws is not None and ws.numel() * ws.element_size() >= 4096 for ws in spaces)
    assert spaces[0].data_ptr() != spaces[1].data_ptr()            # both calls may still be running
    plan.workspace_bytes = 0
    getattr(torch_op, kernel)(x, w)
    assert plan.calls[-1][1] is None


def test_operands_on_different_devices_are_refused(monkeypatch):
    import torch

    from turbofno_b200 import torch_op

    monkeypatch.setattr(torch_op, "_plan", lambda *a, **k: _RecordingPlan(0))
    with pytest.raises(ValueError):
        torch_op._conv1d_cuda(torch.zeros((1, 8, 128), dtype=torch.complex64), torch.zeros((8, 64), dtype=torch.complex64, device="meta"))


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["2d_shared", "1d_per_mode"])
def test_one_shape_on_two_streams_at_once(cuda, kind):
    """Against torch in double precision.  Single-precision transforms of at most 128 x 256 and sums over 64
    channels: eps * log2(n) ~ 6e-8 * 15 and eps * sqrt(64); the parity tolerance of the suite is 1e-5."""
    import torch

    import turbofno_b200.torch_op  # noqa: F401

    signal = (128, 256) if kind == "2d_shared" else (512,)
    B, K, N = (12, 32, 64) if kind == "2d_shared" else (300, 64, 64)
    g = torch.Generator(device="cuda").manual_seed(3)

    def field(*shape):
        return torch.view_as_complex(torch.rand(shape + (2,), generator=g, device="cuda") * 2 - 1)

    def reference(x, w):
        x, w = x.to(torch.complex128), w.to(torch.complex128)
        rank = x.dim() - 2
        kept = (Ellipsis,) + (slice(0, 64),) * rank
        dims = (-2, -1)[-rank:]
        full = torch.zeros((B, N) + signal, dtype=x.dtype, device=x.device)
        full[kept] = torch.einsum("bkxy,kn->bnxy" if w.dim() == 2 else "bkm,knm->bnm", torch.fft.fftn(x, dim=dims)[kept], w)
        return torch.fft.ifftn(full, dim=dims)

    op = torch.ops.turbofno_b200.spectral_conv2d if kind == "2d_shared" else torch.ops.turbofno_b200.spectral_conv1d
    cases = [(field(B, K, *signal), field(K, N, *(() if kind == "2d_shared" else (64,)))) for _ in range(2)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    ys = [[], []]
    for _ in range(6):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                ys[i].append(op(*cases[i]))
    torch.cuda.synchronize()
    for i in range(2):
        ref = reference(*cases[i])
        for y in ys[i]:
            assert ((y - ref).norm() / ref.norm()).item() <= 4e-6
