"""The differentiable convolution at the edges of its block sizes: signals
shorter than a block, than the response, and not a multiple of anything;
responses of 16 and 17 blocks and of more than sixteen parts of the largest
block; rows at odd addresses; recomputed spectra in a workspace that never saw
the forward pass; one gradient alone.  Against float64 (relative L2 <= 1e-6, the
bound of the other gradient tests)."""
import numpy as np
import pytest

from partconv_gb300 import workloads as wl

pytestmark = pytest.mark.gpu

TOL = 1e-6


def _ref(x, h, gy):
    T, L = x.shape[1], len(h)
    y = np.stack([wl.conv_fp64(r, h, T) for r in x])
    gx = np.stack([wl.conv_fp64(g[::-1], h, T)[::-1] for g in gy])
    gh = sum(wl.conv_fp64(g, r[::-1], 2 * T)[T - 1:T - 1 + L] for g, r in zip(gy, x))
    return y, gx, np.concatenate([gh, np.zeros(max(0, L - len(gh)))])


@pytest.mark.parametrize("N,P,B,T,L", [
    ([16], [0], 1, 7, 3), ([16, 64], [4, 0], 3, 100, 400), ([64], [0], 2, 1001, 256), ([128, 1024], [8, 0], 3, 4099, 4096),
    ([128, 1024], [8, 0], 1, 9000, 4097), ([256, 2048], [8, 0], 2, 33000, 20000), ([512, 4096], [8, 0], 3, 50001, 65536),
    ([512, 4096], [8, 0], 1, 70000, 70001), ([1024, 16384], [16, 0], 1, 400000, 300000), ([64], [0], 2, 70, 5000)])
@pytest.mark.parametrize("recompute", [False, True])
def test_sizes(gpu, N, P, B, T, L, recompute):
    import torch

    from partconv_gb300.adjoint import PartitionedConv

    rng = np.random.default_rng(T + L)
    x = (0.1 * rng.standard_normal((B, T))).astype(np.float32)
    h = (0.01 * rng.standard_normal(L)).astype(np.float32)
    gy = rng.standard_normal((B, T)).astype(np.float32)
    mod = PartitionedConv(h, N, P, B, T, recompute=recompute).cuda()
    xd = torch.empty(B * T + 1, device="cuda")[1:].view(B, T).copy_(torch.from_numpy(x)).requires_grad_(True)
    y = mod(xd)
    held = [torch.full((mod.plan.workspace_bytes,), 255, dtype=torch.uint8, device="cuda")]   # the freed workspace's bytes
    gyd = torch.from_numpy(gy).cuda()
    gx, gh = torch.autograd.grad(y, (xd, mod.h), gyd, retain_graph=True)
    del held
    got = [t.detach().cpu().numpy() for t in (y, gx, gh)]
    for a, r in zip(got, _ref(x, h, gy)):
        assert a.shape == r.shape and wl.rel_l2(a, r) <= TOL
    # a second backward pass rebuilds what the first one overwrote; one gradient at a time
    gx2, = torch.autograd.grad(y, (xd,), gyd, retain_graph=True)
    gh2, = torch.autograd.grad(y, (mod.h,), gyd)
    assert np.array_equal(gx2.cpu().numpy(), got[1]) and np.array_equal(gh2.cpu().numpy(), got[2])
