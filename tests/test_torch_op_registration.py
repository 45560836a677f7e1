"""What callers may do with the operators besides calling them: register further kernels and rules, and learn that a
gradient has no derivative of its own."""
import os
import subprocess
import sys

import pytest

from util import ROOT

# in a process of its own: the registrations stay for good
PROGRAM = """
import copy
import torch
from turbofno_b200 import torch_op

def layer(x, w, centered=False):
    dims = (-2, -1)[4 - x.dim():]
    kept = (Ellipsis,) + (slice(0, 64),) * len(dims)
    full = torch.zeros((x.shape[0], w.shape[1]) + x.shape[2:], dtype=x.dtype)
    full[kept] = torch.einsum("bk...,kn->bn...", torch.fft.fftn(x, dim=dims)[kept], w)
    return torch.fft.ifftn(full, dim=dims)

for op, signal in ((torch_op.spectral_conv1d, (128,)), (torch_op.spectral_conv2d, (128, 128))):
    op.register_kernel("cpu", layer)

    @op.register_vmap
    def batch_rule(info, in_dims, x, w, *rest, op=op):
        assert in_dims[:2] == (0, None)
        return op(x.flatten(0, 1), w).unflatten(0, x.shape[:2]), 0

    x, w = torch.randn((3, 2, 8) + signal, dtype=torch.complex64), torch.randn(8, 64, dtype=torch.complex64)
    y = torch.vmap(lambda a: op(a, w))(x)
    assert torch.equal(y, torch.stack([layer(a, w) for a in x]))
    op.register_autocast("cpu", torch.complex64)
    assert "spectral_conv" in repr(op) and op._schema.returns
    # held by a module, copied with it, traced
    assert copy.deepcopy({"op": op})["op"] is op and torch.equal(copy.copy(op)(x[0], w), y[0])
    traced = torch.compile(lambda a, b: op(a, b) * 2, backend="eager", fullgraph=True)
    assert torch.equal(traced(x[0], w), y[0] * 2)
print("ok")
"""


def test_operators_take_further_registrations():
    out = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, capture_output=True, text=True, timeout=300, env=dict(os.environ, PYTHONPATH=ROOT))
    assert out.stdout.strip() == "ok", out.stderr[-2000:]


@pytest.mark.parametrize("which", ["grad_y", "x", "w"])
def test_backward_operator_refuses_to_be_recorded(which):
    import torch

    from turbofno_b200 import torch_op

    t = {"grad_y": torch.zeros((1, 64, 128), dtype=torch.complex64), "x": torch.zeros((1, 64, 128), dtype=torch.complex64),
         "w": torch.zeros((64, 64), dtype=torch.complex64)}
    t[which].requires_grad_(True)
    with pytest.raises(RuntimeError, match="no derivative"):
        torch_op._backward_cuda(t["grad_y"], t["x"], t["w"], False, True, True)


@pytest.mark.gpu
def test_backward_operator_called_directly(cuda):
    import torch

    from test_gpu_backward import _reference, _tensors

    x, w, gy = _tensors(2, 64, 64, (128,), False, False)
    op = torch.ops.turbofno_b200.spectral_conv_backward
    got, want = op(gy, x, w, False, True, True), _reference(x, w, gy, False)[1:]
    for a, b in zip(got, want):
        assert ((a - b).norm() / b.norm()).item() <= 4e-6          # as in the gradient tests
    with pytest.raises(RuntimeError, match="no derivative"):
        op(gy, x.requires_grad_(True), w, False, True, True)
    with torch.no_grad():
        op(gy, x, w, False, True, True)
