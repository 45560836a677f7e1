"""Performance cases of the spectral-convolution layers: what a program that uses this package calls
in earnest, from one short signal to a full image batch, inference and training, complex and real fields.

listed()         the fixed cases
draw(rng)        one more case of the same ranges
prepare(c, s)    what the program holds before the call: plan or weights, inputs made from seed s on the GPU
run(state)       one pass through the public entry points
work(c)          bytes and floating-point operations one pass cannot do without
tolerance(c)     how far another correct single-precision implementation may be off
exact(c, s)      what run returns, from plain torch in double precision
"""
import math

import torch

import turbofno_b200 as tfno
from turbofno_b200 import torch_op

MODES = 64          # retained modes per transformed axis

# Kinds of pass:
#   "plan"   a SpectralConv plan (variant D) called on device tensors, as the drivers and a serving loop do
#   "train"  torch.ops.turbofno_b200.spectral_conv{1,2}d forward, then gradients of input and weights
#   "real"   torch_op.rfft_spectral_conv2d on a real field, inference
#   "real_train"  the same layer, forward and gradients: one FNO training step's share of this layer
# per_mode: one K x N matrix per retained mode (what an FNO layer trains) instead of one shared by all
# modes (what the TurboFNO_{1D,2D}_* grids run).  DX = 0: a 1D layer.
_LARGEST_BYTES = 8 * 128 * 256 * 256 * (64 + 64)


def _case(kind, B, K, N, DY, DX=0, per_mode=False, centered=False, layout="reference", name=None):
    c = {"kind": kind, "B": B, "K": K, "N": N, "DX": DX, "DY": DY, "per_mode": per_mode, "centered": centered, "layout": layout}
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest row of the 1D grid: one signal per channel; latency and launches are everything
        _case("plan", 1, 8, 64, 128, name="1d_one_row"),
        # upper end of the small-batch 1D sweep, wide layer: still far from filling the device
        _case("plan", 64, 32, 128, 256, name="1d_sweep_wide"),
        # an evaluation batch that is a multiple of nothing, channel count between two chunk sizes
        _case("plan", 1003, 40, 64, 256, layout="batch_major", name="1d_ragged"),
        # the large 1D layer the benchmark reports
        _case("plan", 8192, 64, 64, 256, name="1d_large"),
        # long signals, the widest layer of the grid
        _case("plan", 1024, 128, 128, 512, name="1d_long_wide"),
        # a single small image: 2D latency
        _case("plan", 1, 8, 64, 256, DX=128, name="2d_one_image"),
        # the ordinary 2D layer: 16 images, more channels out than in
        _case("plan", 16, 32, 64, 256, DX=256, name="2d_ordinary"),
        # the large 2D layer (one of the chained layers, at the largest batch of the 2D grid)
        _case("plan", 128, 64, 64, 256, DX=256, name="2d_large"),
        # training step of a 1D FNO layer: per-mode weights, forward and both gradients
        _case("train", 512, 64, 64, 512, per_mode=True, layout="batch_major", name="1d_train_per_mode"),
        # training step of a 2D layer with shared weights, odd batch
        _case("train", 7, 64, 64, 128, DX=128, layout="batch_major", name="2d_train_shared"),
        # inference of a 2D FNO layer on a real field: both low-frequency blocks, per-mode weights
        _case("real", 16, 64, 64, 256, DX=256, per_mode=True, centered=True, layout="batch_major", name="2d_real_field"),
        # training step of the same layer on a coarser grid
        _case("real_train", 20, 64, 64, 128, DX=128, per_mode=True, centered=True, layout="batch_major", name="2d_real_train"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    while True:
        kind = rng.choice(["plan", "plan", "plan", "plan", "train", "train", "real", "real_train"])
        two_d = kind.startswith("real") or rng.random() < 0.45
        layout = "batch_major"
        if kind == "plan":
            K, N = 8 * rng.randint(1, 16), rng.choice([64, 64, 128])
            layout = rng.choice(["reference", "batch_major"])
            per_mode = centered = False
            if two_d:
                centered = rng.random() < 0.3
        else:
            # the gradient of the input runs the layer with the channel counts swapped
            per_mode = kind != "train" or rng.random() < 0.6
            K, N = (64, 64) if per_mode else (rng.choice([64, 128]), rng.choice([64, 128]))
            centered = two_d and (kind != "train" or rng.random() < 0.5)
        if two_d:
            c = _case(kind, _log_int(rng, 1, 128), K, N, rng.choice([128, 256]), rng.choice([128, 256]), per_mode, centered, layout)
        else:
            c = _case(kind, _log_int(rng, 1, 8192), K, N, rng.choice([128, 256, 256, 512, 1024]), 0, per_mode, False, layout)
        # no dearer than the largest listed case: a training pass moves and computes about three times
        # what one layer does, and builds whole-field intermediates
        if work(c)["bytes"] <= _LARGEST_BYTES / (1 if kind == "plan" else 4):
            return c


def _uniform(g, shape):
    return torch.view_as_complex(torch.rand(shape + (2,), generator=g, device="cuda").mul_(2).sub_(1))


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    B, K, N, DX, DY = case["B"], case["K"], case["N"], case["DX"], case["DY"]
    signal = (DX, DY) if DX else (DY,)
    modes = (MODES,) * len(signal) if case["per_mode"] else ()
    st = {"kind": case["kind"], "centered": case["centered"]}
    if case["kind"].startswith("real"):
        st["x"] = torch.rand((B, K) + signal, generator=g, device="cuda").mul_(2).sub_(1)
    elif case["layout"] == "reference":
        st["x"] = _uniform(g, (K, B) + signal)
    else:
        st["x"] = _uniform(g, (B, K) + signal)
    wshape = ((N, K) if case["layout"] == "reference" else (K, N)) + modes
    st["w"] = torch.view_as_complex(torch.randn(wshape + (2,), generator=g, device="cuda").mul_(math.sqrt(0.5 / K)))
    if case["kind"] == "plan":
        rank = 2 if DX else 1
        st["plan"] = tfno.SpectralConv(rank, B, DY, K, N, DX=DX or None, variant="D", layout=case["layout"], x_modes_centered=case["centered"])
        st["y"] = torch.empty(st["plan"].out_shape(), dtype=torch.complex64, device="cuda")
    elif case["kind"].endswith("train"):
        st["x"].requires_grad_(True)
        st["w"].requires_grad_(True)
        real = case["kind"] == "real_train"
        st["grad_y"] = torch.rand((B, N) + signal, generator=g, device="cuda").mul_(2).sub_(1) if real else _uniform(g, (B, N) + signal)
    return st


def _layer(st):
    x, w = st["x"], st["w"]
    if st["kind"].startswith("real"):
        return torch_op.rfft_spectral_conv2d(x, w)
    if x.dim() == 3:
        return torch.ops.turbofno_b200.spectral_conv1d(x, w)
    return torch.ops.turbofno_b200.spectral_conv2d(x, w, st["centered"])


def run(state):
    if state["kind"] == "plan":
        return state["plan"](state["x"], state["w"], y=state["y"])
    y = _layer(state)
    if not state["kind"].endswith("train"):
        return y
    grad_x, grad_w = torch.autograd.grad(y, (state["x"], state["w"]), grad_outputs=state["grad_y"])
    return {"y": y.detach(), "grad_x": grad_x, "grad_w": grad_w}


def work(case):
    B, K, N, DX, DY = case["B"], case["K"], case["N"], case["DX"], case["DY"]
    length = (DX or 1) * DY
    modes = MODES * (MODES if DX else 1)
    sample = 4 if case["kind"].startswith("real") else 8
    weights = 8 * K * N * (modes if case["per_mode"] else 1)
    # 5 n log2 n per complex transform (half for a real one), 8 operations per complex multiply-add
    fft = 5 * length * math.log2(length) * (0.5 if sample == 4 else 1.0)
    transforms, contractions = B * (K + N), 1
    data = sample * B * length * (K + N) + weights
    if case["kind"].endswith("train"):
        # backward: read grad_y, write grad_x and grad_w; x and grad_y are transformed once, two
        # contractions (one for each gradient) and one more transform back
        data += sample * B * length * (K + N) + weights
        transforms, contractions = 2 * transforms, 3
    return {"bytes": data, "flops": transforms * fft + contractions * 8.0 * B * K * N * modes}


def tolerance(case):
    # Single-precision transforms and channel sums.  Against the same layer in double precision every
    # case shows a relative error of at most 1.1e-6 and a largest one of 5e-6 of the rms value.
    return {"rel": 4e-6, "max": 2e-5}


def exact(case, seed):
    st = prepare(case, seed)
    reference = case["layout"] == "reference"
    rank = 2 if case["DX"] else 1
    dims = (-2, -1)[-rank:]
    x, w = st["x"].detach(), st["w"].detach().to(torch.complex128)
    if reference:
        x, w = x.transpose(0, 1), w.transpose(0, 1)
    gy = st.get("grad_y")
    grad_w = torch.zeros_like(w)
    ys, gxs = [], []
    # kept modes: 0..63 of every axis, or -32..31 of the first of two
    shift = MODES // 2 if case["centered"] else 0
    step = max(1, 2 ** 26 // (max(x.shape[1], w.shape[1]) * x[0, 0].numel()))
    for b in range(0, x.shape[0], step):
        xb = x[b:b + step].to(torch.float64 if st["kind"].startswith("real") else torch.complex128)
        y, back = _exact_layer(xb, w, dims, shift, None if gy is None else gy[b:b + step])
        ys.append(y)
        if back is not None:
            gxs.append(back[0])
            grad_w += back[1]
    y = torch.cat(ys)
    if gy is not None:
        return {"y": y, "grad_x": torch.cat(gxs), "grad_w": grad_w}
    return y.transpose(0, 1).contiguous() if reference else y


def _exact_layer(x, w, dims, shift, gy):
    length = math.prod(x.shape[2:])
    real = not x.is_complex()
    L = "xy"[-len(dims):]

    def spectrum(t):
        s = torch.fft.fftn(t, dim=dims)
        if shift:
            s = s.roll(shift, dims=-2)
        return s[(Ellipsis,) + (slice(0, MODES),) * len(dims)]

    def field(s):
        full = s.new_zeros(s.shape[:2] + x.shape[2:])
        full[(Ellipsis,) + (slice(0, MODES),) * len(dims)] = s
        if shift:
            full = full.roll(-shift, dims=-2)
        return torch.fft.ifftn(full, dim=dims)

    def mix(spec, mats, sub):
        if mats.dim() == 2:
            sub = sub.replace("%", "")
        return torch.einsum(sub.replace("%", L).replace("#", L), spec, mats)

    # a real field: the kept half spectrum enters the inverse once (ky = 0) or with its mirror image (ky > 0)
    half = torch.ones(MODES, dtype=torch.float64, device=w.device)
    if real:
        half[0] = 0.5
    xs = spectrum(x)
    y = field(mix(xs * half, w, "bk#,kn%->bn#"))
    if real:
        y = 2.0 * y.real
    if gy is None:
        return y, None
    gs = spectrum(gy.to(x.dtype)) * half * (2.0 if real else 1.0)
    grad_x = field(mix(gs, w.conj(), "bn#,kn%->bk#"))
    grad_w = torch.einsum("bk#,bn#->kn%".replace("%", L if w.dim() > 2 else "").replace("#", L), xs.conj(), gs) / length
    return y, (grad_x.real if real else grad_x, grad_w)
