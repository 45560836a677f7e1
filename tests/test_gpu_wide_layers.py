"""Wide 1D layers of long signals: three kernels over the compact spectra when a workspace is given, the fused kernel
when not; both against torch in double precision."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

# tf32 triple products with fp32 accumulation over at most 128 channels and single-precision transforms; the suite's
# parity tolerance is 1e-5
REL = 4e-6


def _layer(x, w, second_forward):
    import torch

    s = torch.einsum("bkm,kn->bnm", torch.fft.fft(x.to(torch.complex128))[..., :64], w.to(torch.complex128))
    s = torch.cat([s, s.new_zeros(s.shape[:2] + (x.shape[-1] - 64,))], -1)
    return torch.fft.fft(s) / x.shape[-1] if second_forward else torch.fft.ifft(s)


def _case(B, K, N, DY, layout, seed=0):
    import torch

    g = torch.Generator(device="cuda").manual_seed(seed + B + K)
    x = torch.view_as_complex(torch.rand((B, K, DY, 2), generator=g, device="cuda") * 2 - 1)
    w = torch.view_as_complex(torch.rand((K, N, 2), generator=g, device="cuda") * 2 - 1)
    if layout == "reference":
        return x, w, x.transpose(0, 1).contiguous(), w.T.contiguous()
    return x, w, x, w


@pytest.mark.parametrize("layout", ["reference", "batch_major"])
@pytest.mark.parametrize("B,K,N,DY", [(148, 8, 128, 512), (301, 128, 128, 1024), (150, 40, 192, 512), (592, 104, 64, 512), (593, 72, 64, 1024)])
@pytest.mark.parametrize("second_forward", [False, True])
def test_both_routes(cuda, B, K, N, DY, layout, second_forward):
    import torch
    import turbofno_b200 as t

    x, w, xm, wm = _case(B, K, N, DY, layout)
    ref = _layer(x, w, second_forward)
    plan = t.SpectralConv(1, B, DY, K, N, layout=layout, second_transform_forward=second_forward, beta=0.5)      # D ignores beta
    assert plan.kernels()[0] == "fft_rows_trunc_kernel<%d>" % (DY // 64) and plan.workspace_bytes > 0
    tiny = torch.empty(16, dtype=torch.uint8, device=cuda)
    for ws in (None, torch.full((plan.workspace_bytes // 4,), float("nan"), device=cuda).view(torch.uint8), tiny):
        y = plan(xm, wm, workspace=ws)
        y = y.transpose(0, 1) if layout == "reference" else y
        err = ((y - ref).norm() / ref.norm()).item()
        assert err <= REL, (ws is None, err)
    # a null workspace through the C interface
    y = torch.full(plan.out_shape(), float("nan"), dtype=torch.complex64, device=cuda)
    ptr = lambda a: ctypes.c_void_p(a.data_ptr())
    assert plan.lib.tfno_exec(plan._plan, ptr(xm), ptr(wm), ptr(y), None, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    y = y.transpose(0, 1) if layout == "reference" else y
    assert ((y - ref).norm() / ref.norm()).item() <= REL
    plan.close()


def test_one_plan_on_two_streams_at_once(cuda):
    """The fused layer shares nothing between calls; with scratch it has to stay so."""
    import torch
    import turbofno_b200 as t

    B, K, N, DY = 300, 64, 128, 512
    plan = t.SpectralConv(1, B, DY, K, N, layout="batch_major")
    cases = [_case(B, K, N, DY, "batch_major", seed) for seed in (1, 2)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    ys = [[], []]
    for _ in range(4):
        for i, s in enumerate(streams):
            if i:
                with torch.cuda.stream(s):
                    ys[i].append(plan(cases[i][0], cases[i][1]))
            else:
                y = torch.empty(plan.out_shape(), dtype=torch.complex64, device=cuda)
                torch.cuda.current_stream().synchronize()
                ys[i].append(plan(cases[i][0], cases[i][1], y=y, stream=s))
    torch.cuda.synchronize()
    for i in range(2):
        ref = _layer(cases[i][0], cases[i][1], False)
        for y in ys[i]:
            assert ((y - ref).norm() / ref.norm()).item() <= REL
    plan.close()


def test_captured_in_a_graph(cuda):
    import torch
    import turbofno_b200 as t

    B, K, N, DY = 160, 16, 128, 512
    x, w, xm, wm = _case(B, K, N, DY, "batch_major")
    plan = t.SpectralConv(1, B, DY, K, N, layout="batch_major")
    y = torch.empty(plan.out_shape(), dtype=torch.complex64, device=cuda)
    plan(xm, wm, y=y)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan(xm, wm, y=y)
    xm.mul_(2.0)
    graph.replay()
    torch.cuda.synchronize()
    ref = _layer(xm, w, False)
    assert ((y - ref).norm() / ref.norm()).item() <= REL
    del graph
    plan.close()
