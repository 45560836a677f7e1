"""What callers may do with the operators besides calling them: register further kernels and rules."""
import os
import subprocess
import sys

from util import ROOT

# in a process of its own: the registrations stay for good
PROGRAM = """
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
print("ok")
"""


def test_operators_take_further_registrations():
    out = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, capture_output=True, text=True, timeout=300, env=dict(os.environ, PYTHONPATH=ROOT))
    assert out.stdout.strip() == "ok", out.stderr[-2000:]
