"""Calls back to back on one stream.  Small launches start beside the tail of the kernel before them; what they read and overwrite
must wait for it all the same.  Long chains, in which every call reads the output of the call before it, share a workspace and see
their weights change in between, against the same chain with a synchronisation after every step, bit for bit."""
import pytest

pytestmark = pytest.mark.gpu

STEPS = 24


def _values(g, shape, real=False):
    import torch

    return torch.rand(shape, generator=g, device="cuda") * 2 - 1 if real else torch.view_as_complex(torch.rand(shape + (2,), generator=g, device="cuda") * 2 - 1)


def _chain(rank, B, sig, per_mode, real, train, step):
    import torch
    import turbofno_b200 as t

    K = N = 64
    g = torch.Generator(device="cuda").manual_seed(5)
    plan = t.SpectralConv(rank, B, sig[-1], K, N, DX=sig[0] if rank == 2 else None, layout="batch_major", per_mode_weights=per_mode)
    a, w = _values(g, (B, K) + sig, real), _values(g, (K, N) + ((64,) * rank if per_mode else ())) * 0.2
    b, gx, gw = torch.empty_like(a), torch.empty_like(a), torch.empty_like(w)
    step()
    seen = []
    for i in range(STEPS):
        plan.exec_real(a, w, y=b) if real else plan(a, w, y=b)
        step()
        if train:
            plan.backward(a, w, b, gx, gw)              # reads the output above, its own workspace from the same pool
            step()
            w.add_(gw / gw.abs().max(), alpha=-1e-3)    # ordinary kernels over what the last one of the library wrote
            step()
            a, gx = gx, a                               # the next call reads grad_x and the one after it overwrites this input
        else:
            w.copy_(w.roll(1, 0))
            step()
            a, b = b, a
        if i % 8 == 7:
            seen += [a.clone(), b.clone(), w.clone(), gw.clone() if train else w]
        if i % 4 == 3:
            a.div_(a.abs().max())
            step()
    torch.cuda.synchronize()
    plan.close()
    return seen


@pytest.mark.parametrize("rank,B,sig,per_mode,real,train", [
    (1, 1, (128,), False, False, False),                # the row-tile kernel alone, one CTA
    (1, 64, (256,), False, False, False),
    (1, 300, (256,), False, False, False),              # the fused kernel
    (2, 1, (128, 128), False, False, False),            # clusters, contraction, parts of an image
    (2, 1, (256, 256), False, False, False),
    (1, 1, (512,), True, False, True),
    (1, 130, (128,), True, False, True),
    (1, 3, (128,), False, False, True),
    (2, 1, (128, 128), False, False, True),
    (2, 1, (128, 256), True, False, True),
    (2, 1, (128, 128), True, True, True),
])
def test_chains_of_calls_equal_the_same_calls_one_at_a_time(cuda, rank, B, sig, per_mode, real, train):
    import torch

    apart = _chain(rank, B, sig, per_mode, real, train, torch.cuda.synchronize)
    assert all(torch.isfinite(torch.view_as_real(v) if v.is_complex() else v).all() for v in apart)
    for _ in range(3):
        together = _chain(rank, B, sig, per_mode, real, train, lambda: None)
        assert all(torch.equal(p, q) for p, q in zip(apart, together))
