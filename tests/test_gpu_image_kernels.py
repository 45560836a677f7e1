"""The whole-image transforms and the per-mode contraction at the edges of their dispatch: few images (a cluster or
several CTAs per image) and many (one CTA, 64-point inverse), both directions, centered modes; row tiles of the
contraction with remainders, and weights whose modes are not adjacent in memory.  Against torch in double precision."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

# single-precision transforms of at most 256 x 256 and sums over at most 72 channels: the error grows like
# eps * log2(n) ~ 6e-8 * 16; the suite's parity tolerance is 1e-5
REL = 2e-6


def _layer(x, w, centered=False, second_forward=False):
    """x[B, K, DX, DY], w[K, N] or w[K, N, 64, 64] -> y[B, N, DX, DY] in double precision."""
    import torch

    x, w = x.to(torch.complex128), w.to(torch.complex128)
    s = torch.fft.fft2(x)
    if centered:
        s = s.roll(32, dims=-2)
    s = torch.einsum("bkxy,kn->bnxy" if w.dim() == 2 else "bkxy,knxy->bnxy", s[..., :64, :64], w)
    full = torch.zeros(s.shape[:2] + x.shape[2:], dtype=s.dtype, device=s.device)
    full[..., :64, :64] = s
    if centered:
        full = full.roll(-32, dims=-2)
    return torch.fft.fft2(full) / (x.shape[2] * x.shape[3]) if second_forward else torch.fft.ifft2(full)


def _check(y, ref):
    err = ((y - ref).norm() / ref.norm()).item()
    assert err <= REL, err


def _field(g, *shape):
    import torch

    return torch.view_as_complex(torch.rand(shape + (2,), generator=g, device="cuda") * 2 - 1)


@pytest.mark.parametrize("DX,DY", [(128, 128), (128, 256), (256, 128), (256, 256)])
@pytest.mark.parametrize("B", [1, 3, 10])            # 8 .. 80 input and 64 .. 640 output images: both sides of every threshold
@pytest.mark.parametrize("mode", ["corner", "centered", "second_forward"])
def test_image_transforms_few_and_many_images(cuda, DX, DY, B, mode):
    import torch
    import turbofno_b200 as t

    g = torch.Generator(device="cuda").manual_seed(B)
    for K in (8, 40):
        x, w = _field(g, B, K, DX, DY), _field(g, K, 64)
        plan = t.SpectralConv(2, B, DY, K, 64, DX=DX, layout="batch_major", x_modes_centered=mode == "centered",
                              second_transform_forward=mode == "second_forward")
        _check(plan(x, w), _layer(x, w, mode == "centered", mode == "second_forward"))
        plan.close()


@pytest.mark.parametrize("rows", [1, 4, 5, 8, 9, 12, 13, 16, 17, 24, 25, 32, 33, 49])
def test_per_mode_contraction_row_tiles(cuda, rows):
    import torch
    import turbofno_b200 as t

    g = torch.Generator(device="cuda").manual_seed(rows)
    K, N, DY = (72 if rows % 2 else 8), (128 if rows in (1, 33) else 64), 128
    x, w = _field(g, rows, K, DY), _field(g, K, N, 64)
    plan = t.SpectralConv(1, rows, DY, K, N, layout="batch_major", per_mode_weights=True)
    s = torch.einsum("bkm,knm->bnm", torch.fft.fft(x.to(torch.complex128))[..., :64], w.to(torch.complex128))
    _check(plan(x, w), torch.fft.ifft(torch.cat([s, s.new_zeros(rows, N, DY - 64)], -1)))
    plan.close()


@pytest.mark.parametrize("order", ["mkn", "nmk", "odd"])
def test_per_mode_weights_in_other_orders(cuda, order):
    """Mode stride other than 1, or odd strides: the weights travel one mode at a time."""
    import torch
    import turbofno_b200 as t
    from turbofno_b200._lib import Problem, check, load

    B, K, N, DY = 7, 16, 64, 128
    g = torch.Generator(device="cuda").manual_seed(2)
    x, w = _field(g, B, K, DY), _field(g, K, N, 64)
    if order == "mkn":
        mem, strides = w.permute(2, 0, 1).contiguous(), (N, 1, K * N)
    elif order == "nmk":
        mem, strides = w.permute(1, 2, 0).contiguous(), (1, 64 * K, K)
    else:
        mem = torch.zeros((K, N, 65), dtype=torch.complex64, device=cuda)
        mem[..., :64] = w
        strides = (N * 65, 65, 1)
    lib, handle = load(), t.Handle.get(0)
    p = Problem()
    check(lib.tfno_problem_init(ctypes.byref(p), 1))
    p.bs, p.DY, p.K, p.N = B, DY, K, N
    p.x_stride_b, p.x_stride_k, p.y_stride_b, p.y_stride_n = K * DY, DY, N * DY, DY
    p.w_stride_k, p.w_stride_n, p.w_stride_m = strides
    plan = ctypes.c_void_p()
    check(lib.tfno_plan_create(handle._h, ctypes.byref(p), ctypes.byref(plan)))
    ws = torch.empty(lib.tfno_workspace_bytes(plan), dtype=torch.uint8, device=cuda)
    y = torch.empty((B, N, DY), dtype=torch.complex64, device=cuda)
    ptr = lambda a: ctypes.c_void_p(a.data_ptr())
    check(lib.tfno_exec(plan, ptr(x), ptr(mem), ptr(y), ptr(ws), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    torch.cuda.synchronize()
    lib.tfno_plan_destroy(plan)
    s = torch.einsum("bkm,knm->bnm", torch.fft.fft(x.to(torch.complex128))[..., :64], w.to(torch.complex128))
    _check(y, torch.fft.ifft(torch.cat([s, s.new_zeros(B, N, DY - 64)], -1)))


@pytest.mark.parametrize("DX,DY", [(128, 128), (128, 256), (256, 128), (256, 256)])
@pytest.mark.parametrize("images", [152, 200, 296, 304, 320])       # just above a wave of images, two thirds of one, a full one
@pytest.mark.parametrize("real", [False, True])
def test_forward_images_around_the_waves_of_a_launch(cuda, DX, DY, images, real):
    """One CTA or a cluster of them per image, by how much of the last wave would stay empty."""
    import torch
    import turbofno_b200 as t

    g = torch.Generator(device="cuda").manual_seed(images)
    K, B = 8, images // 8
    plan = t.SpectralConv(2, B, DY, K, 64, DX=DX, layout="batch_major", per_mode_weights=real, x_modes_centered=real)
    if real:
        x, w = torch.rand((B, K, DX, DY), generator=g, device="cuda") * 2 - 1, _field(g, K, 64, 64, 64)
        half = torch.ones(64, dtype=torch.float64, device="cuda")
        half[0] = 0.5
        _check(plan.exec_real(x, w), 2 * _layer(x, w.to(torch.complex128) * half, True).real)
    else:
        x, w = _field(g, B, K, DX, DY), _field(g, K, 64)
        _check(plan(x, w), _layer(x, w))
    plan.close()


@pytest.mark.parametrize("DX,DY", [(128, 128), (256, 128), (256, 256)])
@pytest.mark.parametrize("B", [1, 5])                # a cluster and one CTA per image
@pytest.mark.parametrize("pad_channel,pad_batch", [(2, 0), (0, 2), (6, 4), (4, 0)])
def test_real_images_apart_by_any_even_number_of_samples(cuda, DX, DY, B, pad_channel, pad_batch):
    """Layer and gradients of real images with gaps between them: those that start on 8-byte boundaries only, too.  Bit for bit
    the results of dense images, and the gaps stay as they are."""
    import torch
    import turbofno_b200 as t
    from turbofno_b200._lib import Problem, check, load

    K = N = 64
    g = torch.Generator(device="cuda").manual_seed(3)
    real = lambda: torch.rand((B, K, DX, DY), generator=g, device="cuda") * 2 - 1
    x, gy, w = real(), real(), _field(g, K, N, 64, 64)
    dense = t.SpectralConv(2, B, DY, K, N, DX=DX, layout="batch_major", per_mode_weights=True, x_modes_centered=True)
    want = [dense.exec_real(x, w), torch.empty_like(x), torch.empty_like(w)]
    dense.backward(x, w, gy, want[1], want[2])
    dense.close()

    stride_k = DX * DY + pad_channel
    stride_b = K * stride_k + pad_batch

    def apart(values=None):
        mem = torch.full((B * stride_b,), 7.0, device=cuda)
        view = mem.as_strided((B, K, DX, DY), (stride_b, stride_k, DY, 1))
        if values is not None:
            view.copy_(values)
        return mem, view

    lib, handle = load(), t.Handle.get(0)
    p = Problem()
    check(lib.tfno_problem_init(ctypes.byref(p), 2))
    p.bs, p.DX, p.DY, p.K, p.N, p.x_modes_centered = B, DX, DY, K, N, 1
    p.x_stride_b = p.y_stride_b = stride_b
    p.x_stride_k = p.y_stride_n = stride_k
    p.w_stride_k, p.w_stride_n, p.w_stride_m = N * 4096, 4096, 1
    plan = ctypes.c_void_p()
    check(lib.tfno_plan_create(handle._h, ctypes.byref(p), ctypes.byref(plan)))
    ws = torch.empty(max(lib.tfno_workspace_bytes(plan), lib.tfno_backward_workspace_bytes(plan)), dtype=torch.uint8, device=cuda)
    (xm, _), (gym, _), (ym, y), (gxm, gx) = apart(x), apart(gy), apart(), apart()
    gw = torch.empty_like(w)
    stream = torch.cuda.current_stream().cuda_stream
    check(lib.tfno_exec_real(plan, xm.data_ptr(), w.data_ptr(), ym.data_ptr(), ws.data_ptr(), stream))
    check(lib.tfno_backward(plan, 1, xm.data_ptr(), w.data_ptr(), gym.data_ptr(), gxm.data_ptr(), gw.data_ptr(), ws.data_ptr(), stream))
    torch.cuda.synchronize()
    lib.tfno_plan_destroy(plan)
    for got, ref in ((y, want[0]), (gx, want[1]), (gw, want[2])):
        assert torch.equal(got, ref)
    for mem, view in ((ym, y), (gxm, gx)):
        view.fill_(7.0)
        assert (mem == 7.0).all()
