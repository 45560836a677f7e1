"""Scratch that wide 1D layers can do without: tfno_exec needs none and leaves a workspace alone, tfno_exec_scratch uses
what is large enough, and the host-buffer path does not ask for it."""
import ctypes
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

REL = 4e-6          # as in the wide-layer tests: tf32 triple products over at most 128 channels, single-precision transforms


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _inputs(B, K, N, DY):
    """x[B, K, DY], w[K, N] and the layer in double precision."""
    import torch

    g = torch.Generator(device="cuda").manual_seed(B)
    x = torch.view_as_complex(torch.rand((B, K, DY, 2), generator=g, device="cuda") * 2 - 1)
    w = torch.view_as_complex(torch.rand((K, N, 2), generator=g, device="cuda") * 2 - 1)
    s = torch.einsum("bkm,kn->bnm", torch.fft.fft(x.to(torch.complex128))[..., :64], w.to(torch.complex128))
    return x, w, torch.fft.ifft(torch.cat([s, s.new_zeros(B, N, DY - 64)], -1))


def _sizes(plan):
    return plan.lib.tfno_workspace_bytes(plan._plan), plan.lib.tfno_optional_workspace_bytes(plan._plan)


# (rows, K, N, DY) -> has optional scratch, for 148 SMs
@pytest.mark.parametrize("B,K,N,DY,offered", [
    (148, 8, 128, 512, True), (147, 8, 128, 512, False), (148, 8, 128, 256, False), (300, 136, 128, 512, False),
    (592, 104, 64, 512, True), (591, 104, 64, 512, False), (592, 96, 64, 512, False), (592, 64, 64, 1024, True), (592, 56, 64, 1024, False)])
def test_what_is_needed_and_what_is_offered(cuda, B, K, N, DY, offered):
    import turbofno_b200 as t

    assert t.Handle.get(0).sm_count == 148
    plan = t.SpectralConv(1, B, DY, K, N)
    spectra = sum((8 * 64 * B * c + 255) // 256 * 256 for c in (K, N))
    assert _sizes(plan) == (0, spectra if offered else 0)
    plan.close()


def test_plans_that_need_scratch_offer_none(cuda):
    import turbofno_b200 as t

    for plan in (t.SpectralConv(2, 2, 128, 8, 64), t.SpectralConv(1, 300, 512, 64, 128, variant="A"),
                 t.SpectralConv(1, 300, 512, 64, 128, per_mode_weights=True)):
        need, offer = _sizes(plan)
        assert need > 0 and offer == 0 and plan.workspace_bytes == need
        assert plan.lib.tfno_exec_scratch(plan._plan, *[ctypes.c_void_p(1 << 20)] * 4, need - 1, None) == t._lib.ERR_WORKSPACE
        plan.close()


def test_tfno_exec_leaves_the_workspace_alone(cuda):
    """One buffer given to calls on two streams at once: none of them may use it."""
    import torch
    import turbofno_b200 as t

    B, K, N, DY = 300, 32, 128, 512
    x, w, ref = _inputs(B, K, N, DY)
    plan = t.SpectralConv(1, B, DY, K, N, layout="batch_major")
    ws = torch.full((plan.workspace_bytes,), 0x5a, dtype=torch.uint8, device=cuda)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    ys = [torch.empty_like(ref, dtype=torch.complex64) for _ in range(4)]
    torch.cuda.synchronize()
    for i, y in enumerate(ys):
        assert plan.lib.tfno_exec(plan._plan, _ptr(x), _ptr(w), _ptr(y), _ptr(ws), ctypes.c_void_p(streams[i % 2].cuda_stream)) == 0
    torch.cuda.synchronize()
    assert (ws == 0x5a).all()
    for y in ys:
        assert ((y - ref).norm() / ref.norm()).item() <= REL
    # too little of it: as without
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    for nbytes, untouched in ((plan.workspace_bytes - 1, True), (plan.workspace_bytes, False)):
        y = torch.empty_like(ys[0])
        assert plan.lib.tfno_exec_scratch(plan._plan, _ptr(x), _ptr(w), _ptr(y), _ptr(ws), nbytes, st) == 0
        torch.cuda.synchronize()
        assert (ws == 0x5a).all().item() == untouched
        assert ((y - ref).norm() / ref.norm()).item() <= REL
    plan.close()


def test_host_path_does_not_ask_for_it(cuda):
    """exec_host keeps two chunks of x, y and w on the device and nothing else."""
    import torch
    import turbofno_b200 as t

    B, K, N, DY = 512, 8, 128, 512
    x, w, ref = _inputs(B, K, N, DY)
    xh, wh = x.transpose(0, 1).contiguous().cpu(), w.T.contiguous().cpu()
    yh = torch.empty((N, B, DY), dtype=torch.complex64)
    warm = t.SpectralConv(1, B, DY, K, N)                       # kernels of both routes are on the device from here on
    y = torch.empty(warm.out_shape(), dtype=torch.complex64, device=cuda)
    warm(x.transpose(0, 1).contiguous(), w.T.contiguous(), y=y)
    assert warm.lib.tfno_exec(warm._plan, _ptr(x), _ptr(w), _ptr(y), None, None) == 0
    plan = t.SpectralConv(1, B, DY, K, N)
    plan.set_host_chunk(B)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    plan.exec_host(xh, wh, yh)
    used = before - torch.cuda.mem_get_info()[0]
    staging = 2 * 8 * (B * DY * (K + N) + K * N)
    assert plan.workspace_bytes > 32 << 20 and used < staging + plan.workspace_bytes, (used, staging)
    assert ((yh.transpose(0, 1).to(cuda) - ref).norm() / ref.norm()).item() <= REL
    plan.close()
    warm.close()


def test_executable_runs_a_wide_layer(cuda):
    import json

    from test_gpu_drivers import BIN

    out = subprocess.check_output([os.path.join(BIN, "TurboFNO_1D_D"), "300", "1", "1024", "128", "128", "--stream", "--json"], text=True, timeout=120)
    assert json.loads(out)["time_ms"] > 0, out


def test_a_captured_call_records_no_block_of_the_allocator(cuda):
    """A graph may be captured by other means than torch.cuda.graph, whose pool would keep the block; with a workspace
    the graph uses that."""
    import torch
    import turbofno_b200 as t

    B, K, N, DY = 160, 16, 128, 512
    x, w, ref = _inputs(B, K, N, DY)
    plan = t.SpectralConv(1, B, DY, K, N, layout="batch_major")
    y = torch.empty(plan.out_shape(), dtype=torch.complex64, device=cuda)
    ws = torch.empty(plan.workspace_bytes, dtype=torch.uint8, device=cuda)
    side = torch.cuda.Stream()
    for kw in ({}, {"workspace": ws}, {"stream": side}):
        plan(x, w, y=y, **kw)
        torch.cuda.synchronize()
        y.zero_()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            before = torch.cuda.memory_stats()["allocation.all.allocated"]
            plan(x, w, y=y, **kw)
            allocated = torch.cuda.memory_stats()["allocation.all.allocated"] - before
        assert allocated == 0, kw
        graph.replay()
        torch.cuda.synchronize()
        assert ((y - ref).norm() / ref.norm()).item() <= REL
        del graph
    plan.close()
