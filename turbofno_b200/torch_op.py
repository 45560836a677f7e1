"""PyTorch operators `torch.ops.turbofno_b200.spectral_conv1d / spectral_conv2d` over the C ABI.

For callers that hold activations the PyTorch way, batch first:

    spectral_conv1d(x[B, K, DY], w[K, N]) -> y[B, N, DY]
    spectral_conv2d(x[B, K, DX, DY], w[K, N], x_modes_centered=False) -> y[B, N, DX, DY]

complex64, CUDA, contiguous; 64 kept modes per transformed axis (the corner block in 2D), weights
shared by all modes, unnormalised forward and 1/DY (1/(DX*DY)) inverse transform -- the layer the
reference's fully fused variant D computes (fusion_variants/1D_D_exp_fused_fft_cgemm_ifft/,
fusion_variants/2D_D_exp_fused_fft_cgemm_ifft/), which has no framework binding of its own.

Beyond the reference, for callers that train an FNO:

  * per-mode weights: w[K, N, 64] (1D) or w[K, N, 64, 64] (2D), one K x N matrix per kept mode;
  * x_modes_centered (2D): X index i of the kept block is frequency i - 32, i.e. both low-frequency
    blocks of the non-last axis (rows 32..63 are what FNO code calls weights1, kx = 0..31; rows
    0..31 are weights2, kx = -32..-1);
  * rfft_spectral_conv2d(x_real, w): the rfft2 -> weights -> irfft2 layer of a real-valued field,
    on image kernels that read and write real samples (see the function).

The operators are registered with torch.library, so they carry a shape function for tracing and
export; they run on the caller's current stream and allocate their results and scratch through the
caching allocator.  Plans are cached per (shape, device).

The operators have autograd formulas built from the same kernels: the layer is
y = A(x) W with A = (1/DY) F^H P F (P keeps 64 modes), A is self-adjoint, so
grad_x is the layer of grad_y with W^H -- which needs the kernel's shape limits for the swapped
channel counts (K a multiple of 64, N a multiple of 8) -- and grad_W = X^H G / DY per mode, summed
over the batch and (for weights shared by all modes) over the modes, with X, G the truncated spectra of
x and grad_y.  The same holds in two dimensions with 1/(DX*DY).
"""
import torch

from . import api

_plans = {}


def _plan(rank, bs, DY, K, N, DX, device, per_mode=False, centered=False):
    key = (rank, bs, DY, K, N, DX, device, per_mode, centered)
    plan = _plans.get(key)
    if plan is None:
        plan = api.SpectralConv(rank, bs, DY, K, N, DX=DX, variant="D", layout="batch_major", device=device,
                                per_mode_weights=per_mode, x_modes_centered=centered)
        _plans[key] = plan
    return plan


def _run_layer(plan, x, w, y):
    """One layer with scratch of its own.  Every caller of a shape shares its plan, on any stream and thread, and the
    plan's own buffer serves one stream and one thread at a time: two calls in flight would write the same spectra.
    The plan is made from the shapes of x and w, whose types the operator has checked."""
    if w.device != x.device:
        raise ValueError("w is on %s, x on %s" % (w.device, x.device))
    return plan._launch(x, w, y, plan.call_scratch(x.device))


def _check(x, w, rank):
    """Returns True when w carries one matrix per mode."""
    if x.dtype != torch.complex64 or w.dtype != torch.complex64:
        raise TypeError("spectral_conv%dd: x and w must be complex64" % rank)
    per_mode = w.dim() == 2 + rank
    if x.dim() != rank + 2 or not (w.dim() == 2 or per_mode) or w.shape[0] != x.shape[1] or \
            (per_mode and tuple(w.shape[2:]) != (64,) * rank):
        raise ValueError("spectral_conv%dd: expected x[B, K%s, DY] and w[K, N] or w[K, N%s]" %
                         (rank, ", DX" if rank == 2 else "", ", 64" * rank))
    return per_mode


# Defined through torch.library's Library: schema, CUDA kernel, shape function and autograd formula, without the checks
# that custom_op's wrapper makes around every call of the kernel.
_lib = torch.library.Library("turbofno_b200", "FRAGMENT")


def _define(schema, kernel, fake):
    name = schema[:schema.index("(")]
    _lib.define(schema, tags=torch.Tag.pt2_compliant_tag)
    _lib.impl(name, kernel, "CUDA")
    torch.library.register_fake("turbofno_b200::" + name, fake, lib=_lib)
    return getattr(torch.ops.turbofno_b200, name).default


class _Operator:
    """An operator as callers of this module hold it: called like a function, and open to the registrations that
    torch.library offers for custom operators."""

    def __init__(self, overload):
        self._overload = overload

    def __call__(self, *args, **kwargs):
        return self._overload(*args, **kwargs)

    def __getattr__(self, name):
        if name == "_overload":                     # a copy in the making
            raise AttributeError(name)
        return getattr(self._overload, name)

    def __deepcopy__(self, memo):
        return self

    def __repr__(self):
        return "<operator %s>" % self._overload.name()

    def register_kernel(self, device_types, func=None):
        return torch.library.register_kernel(self._overload, device_types, func)

    def register_fake(self, func):
        return torch.library.register_fake(self._overload, func, allow_override=True)

    def register_autocast(self, device_type, cast_inputs):
        return torch.library.register_autocast(self._overload, device_type, cast_inputs)

    def register_vmap(self, func=None):
        return torch.library.register_vmap(self._overload, func)

    def register_torch_dispatch(self, torch_dispatch_class, func=None):
        return torch.library.register_torch_dispatch(self._overload, torch_dispatch_class, func)


def _differentiable(name, backward, setup_context):
    torch.library.register_autograd("turbofno_b200::" + name, backward, setup_context=setup_context, lib=_lib)


def _conv1d_cuda(x, w):
    per_mode = _check(x, w, 1)
    x, w = x.contiguous(), w.contiguous()
    B, K, DY = x.shape
    N = w.shape[1]
    plan = _plan(1, B, DY, K, N, None, x.device.index, per_mode)
    return _run_layer(plan, x, w, torch.empty((B, N, DY), dtype=torch.complex64, device=x.device))


def _conv1d_fake(x, w):
    _check(x, w, 1)
    return x.new_empty((x.shape[0], w.shape[1], x.shape[2]))


spectral_conv1d = _Operator(_define("spectral_conv1d(Tensor x, Tensor w) -> Tensor", _conv1d_cuda, _conv1d_fake))


def _conv2d_cuda(x, w, x_modes_centered=False):
    per_mode = _check(x, w, 2)
    x, w = x.contiguous(), w.contiguous()
    B, K, DX, DY = x.shape
    N = w.shape[1]
    plan = _plan(2, B, DY, K, N, DX, x.device.index, per_mode, bool(x_modes_centered))
    return _run_layer(plan, x, w, torch.empty((B, N, DX, DY), dtype=torch.complex64, device=x.device))


def _conv2d_fake(x, w, x_modes_centered=False):
    _check(x, w, 2)
    return x.new_empty((x.shape[0], w.shape[1], x.shape[2], x.shape[3]))


spectral_conv2d = _Operator(_define("spectral_conv2d(Tensor x, Tensor w, bool x_modes_centered=False) -> Tensor", _conv2d_cuda, _conv2d_fake))


def _truncated_spectrum(t):
    """[B, C, DY] -> [B, C, 64]: forward transform of every signal, first 64 modes (tfno_fft_stride_DY)."""
    B, C, DY = t.shape
    out = torch.empty((B, C, 64), dtype=torch.complex64, device=t.device)
    api.fft_stride_DY(t.contiguous(), out, B * C, DY)
    return out


# ---- gradients ---------------------------------------------------------------------------------
# One call of the library computes both (tfno_backward): the spectrum of grad_y serves grad_x and grad_w.  It has no
# gradient of its own, so a backward pass that is itself recorded (create_graph) takes the formulas below
# it, whose grad_x is made of the differentiable operators; so do channel counts beyond _NATIVE_CHANNELS: 192 is as far as
# the tensor-core kernels and the gradient tests go, not a line of speed (1D, 64 rows, DY = 256: 159 against 232 us with
# the formulas at 192 channels, 249 against 327 at 256).
_NATIVE_CHANNELS = 192


def _aligned(t):
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


def _backward_cuda(grad_y, x, w, x_modes_centered, need_x, need_w):
    if torch.is_grad_enabled() and (grad_y.requires_grad or x.requires_grad or w.requires_grad):
        raise RuntimeError("spectral_conv_backward has no derivative formula: differentiate the layer with create_graph=True")
    rank = x.dim() - 2
    grad_y, x, w = _aligned(grad_y), _aligned(x), _aligned(w)
    plan = _plan(rank, x.shape[0], x.shape[-1], x.shape[1], w.shape[1], x.shape[2] if rank == 2 else None, x.device.index,
                 w.dim() > 2, x_modes_centered)
    grad_x = torch.empty_like(x) if need_x else x.new_empty(0)
    grad_w = torch.empty_like(w) if need_w else w.new_empty(0)
    if need_x or need_w:
        plan.backward(x, w, grad_y, grad_x if need_x else None, grad_w if need_w else None)
    return grad_x, grad_w


def _backward_fake(grad_y, x, w, x_modes_centered, need_x, need_w):
    return (torch.empty_like(x, memory_format=torch.contiguous_format) if need_x else x.new_empty(0),
            torch.empty_like(w, memory_format=torch.contiguous_format) if need_w else w.new_empty(0))


spectral_conv_backward = _define("spectral_conv_backward(Tensor grad_y, Tensor x, Tensor w, bool x_modes_centered, bool need_x, bool need_w) -> (Tensor, Tensor)",
                                 _backward_cuda, _backward_fake)


def _native_backward(ctx, grad_y, centered):
    """(grad_x, grad_w), or None when the differentiable formulas have to be taken."""
    x, w = ctx.saved_tensors
    if torch.is_grad_enabled() or max(w.shape[0], w.shape[1]) > _NATIVE_CHANNELS:
        return None
    need_x, need_w = ctx.needs_input_grad[0], ctx.needs_input_grad[1]
    grad_x, grad_w = spectral_conv_backward(grad_y, x, w, centered, need_x, need_w)
    return (grad_x if need_x else None), (grad_w if need_w else None)


def _conv1d_setup_context(ctx, inputs, output):
    x, w = inputs
    ctx.save_for_backward(x, w)


def _conv2d_setup_context(ctx, inputs, output):
    x, w, centered = inputs
    ctx.save_for_backward(x, w)
    ctx.centered = bool(centered)


def _conv1d_backward(ctx, grad_y):
    native = _native_backward(ctx, grad_y, False)
    if native is not None:
        return native
    x, w = ctx.saved_tensors
    grad_x = grad_w = None
    grad_y = grad_y.contiguous()
    if ctx.needs_input_grad[0]:
        grad_x = spectral_conv1d(grad_y, w.conj().transpose(0, 1).contiguous())
    if ctx.needs_input_grad[1]:
        X, G = _truncated_spectrum(x), _truncated_spectrum(grad_y)
        grad_w = torch.einsum("bkm,bnm->knm" if w.dim() == 3 else "bkm,bnm->kn", X.conj(), G) / x.shape[2]
    return grad_x, grad_w


_differentiable("spectral_conv1d", _conv1d_backward, _conv1d_setup_context)


def _truncated_spectrum2d(t, centered=False):
    """[B, C, DX, DY] -> [B, C, 64, 64]: X transform keeping 64 modes (tfno_fft_stride), then Y.
    Centered X modes are the first 64 modes of the field multiplied by exp(2 pi i 32 x / DX)."""
    B, C, DX, DY = t.shape
    if centered:
        turns = (torch.arange(DX, device=t.device) * 32 % DX).to(torch.float64) / DX      # reduced before the sine
        phase = torch.polar(torch.ones(DX, dtype=torch.float64, device=t.device), 2 * torch.pi * turns)
        t = t * phase.to(torch.complex64)[:, None]
    tx = torch.empty((B, C, 64, DY), dtype=torch.complex64, device=t.device)
    api.fft_stride(t.contiguous(), tx, DY, B * C * DY, DX)
    out = torch.empty((B, C, 64, 64), dtype=torch.complex64, device=t.device)
    api.fft_stride_DY(tx, out, B * C * 64, DY)
    return out


def _conv2d_backward(ctx, grad_y):
    native = _native_backward(ctx, grad_y, ctx.centered)
    if native is not None:
        return native + (None,)
    x, w = ctx.saved_tensors
    grad_x = grad_w = None
    grad_y = grad_y.contiguous()
    if ctx.needs_input_grad[0]:
        grad_x = spectral_conv2d(grad_y, w.conj().transpose(0, 1).contiguous(), ctx.centered)
    if ctx.needs_input_grad[1]:
        X, G = _truncated_spectrum2d(x, ctx.centered), _truncated_spectrum2d(grad_y, ctx.centered)
        grad_w = torch.einsum("bkxy,bnxy->knxy" if w.dim() == 4 else "bkxy,bnxy->kn", X.conj(), G) / (x.shape[2] * x.shape[3])
    return grad_x, grad_w, None


_differentiable("spectral_conv2d", _conv2d_backward, _conv2d_setup_context)


def _real_conv2d_cuda(x, w):
    _check_real(x, w)
    x, w = _aligned(x), _aligned(w)
    B, K, DX, DY = x.shape
    plan = _plan(2, B, DY, K, w.shape[1], DX, x.device.index, True, True)
    return plan.exec_real(x, w)


def _check_real(x, w):
    if x.dtype != torch.float32 or w.dtype != torch.complex64:
        raise TypeError("rfft_spectral_conv2d: x must be float32 and w complex64")
    if x.dim() != 4 or w.shape[0] != x.shape[1] or tuple(w.shape[2:]) != (64, 64):
        raise ValueError("rfft_spectral_conv2d: expected x[B, K, DX, DY] and w[K, N, 64, 64]")


def _real_conv2d_fake(x, w):
    _check_real(x, w)
    return x.new_empty((x.shape[0], w.shape[1], x.shape[2], x.shape[3]))


real_spectral_conv2d = _define("real_spectral_conv2d(Tensor x, Tensor w) -> Tensor", _real_conv2d_cuda, _real_conv2d_fake)


def _real_conv2d_setup_context(ctx, inputs, output):
    x, w = inputs
    ctx.save_for_backward(x, w)


def _real_conv2d_backward(ctx, grad_y):
    native = _native_backward(ctx, grad_y, True)
    if native is not None:
        return native
    # the layer's adjoint has its own form; grad_w: factors 1 at ky = 0 and 2 elsewhere
    x, w = ctx.saved_tensors
    grad_x = grad_w = None
    if ctx.needs_input_grad[0]:
        grad_x = real_spectral_conv2d(grad_y, w.conj().transpose(0, 1).contiguous())
    if ctx.needs_input_grad[1]:
        X, G = (_truncated_spectrum2d(torch.complex(t, torch.zeros_like(t)), True) for t in (x, grad_y))
        twice = torch.full((64,), 2.0, dtype=torch.float32, device=w.device)
        twice[0] = 1.0
        grad_w = torch.einsum("bkxy,bnxy->knxy", X.conj(), G) * (twice / (x.shape[2] * x.shape[3]))
    return grad_x, grad_w


_differentiable("real_spectral_conv2d", _real_conv2d_backward, _real_conv2d_setup_context)


def rfft_spectral_conv2d(x, w):
    """The spectral layer of a real-valued field as FNO code writes it,

        irfft2(pad(einsum("bkxy,knxy->bnxy", rfft2(x)[:, :, kx, :64], w)), s=(DX, DY)),  kx = -32..31,

    for real x[B, K, DX, DY] (float32) and per-mode weights w[K, N, 64, 64] (complex64, X index i is
    frequency i - 32).  The real inverse transform of a half spectrum Z is 2 Re(ifft2(Z')) with Z' = Z
    except for the ky = 0 column, which enters once and is halved; the image kernels read and write real
    samples and transform two rows in one complex transform.
    irfft2 here means the complex inverse along X followed by a real inverse along Y that drops the
    imaginary part of the ky = 0 bin (torch on the CPU); free weights leave a complex value there,
    for which torch's CUDA backend returns something else.
    Differentiable in x and w."""
    if x.is_complex() or w.dim() != 4:
        raise ValueError("rfft_spectral_conv2d: expected real x[B, K, DX, DY] and w[K, N, 64, 64]")
    return real_spectral_conv2d(x.to(torch.float32), w)
