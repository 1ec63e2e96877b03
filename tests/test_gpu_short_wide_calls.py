"""Block-parallel calls shorter than the larger levels' blocks: the partial sums of
a block in progress are built by several calls and one-block steps in turn, each a
part.  The same bits as one call (MIMO: within 1e-5 of float64), for levels that
fire within their step, deferred ones, several base blocks per step and handles
whose many tiles move the line where such calls begin."""
import numpy as np
import pytest

from partconv_gb300 import PC_PLANAR, PartConvMulti
from partconv_gb300 import workloads as wl
from partconv_gb300.mimo import PartConvMIMO

pytestmark = pytest.mark.gpu


def _cut(m, x, sizes):
    """planar device calls of the given numbers of blocks, again and again"""
    import torch

    B, n = m.buffer_size, x.shape[1]
    out, at, i = [], 0, 0
    while at < n:
        k = min(sizes[i % len(sizes)] * B, n - at)
        xi = x[:, at:at + k].contiguous()
        y = torch.empty(m.numOutputChannels, k, device="cuda")
        m.process_device(y, xi, k, PC_PLANAR)
        out.append(y)
        at, i = at + k, i + 1
    torch.cuda.synchronize()
    return torch.cat(out, 1).cpu().numpy()


@pytest.mark.parametrize("n,N,P,L,K", [
    (1, [16, 1024], [64, 0], 20000, 1), (1, [64, 16384], [256, 0], 70000, 1),        # in-step: s_L = N_L
    (2, [16, 512], [70, 0], 12000, 1), (2, [64, 256, 4096], [8, 40, 0], 40000, 1),   # deferred
    (1, [64, 2048], [32, 0], 50000, 1), (1, [32, 65536], [2048, 0], 200000, 1),
    (2, [64, 4096], [70, 0], 60000, 2), (2, [64, 4096], [64, 0], 60000, 4),
    (40, [64, 16384], [257, 0], 40000, 1), (12, [16, 64, 256, 1024, 4096, 16384, 65536], [4, 3, 3, 3, 3, 3, 0], 150000, 1)])
def test_partial_sums_over_several_calls(gpu, n, N, P, L, K):
    import torch

    rng = np.random.default_rng(L + n)
    pcs = [dict(ir=wl.decaying_ir(rng, L - 11 * c, 0.3), N=N, P=P, in_ch=c, out_ch=c) for c in range(n)]
    blocks = min(max(700, 3 * N[-1] // N[0] + L // N[0]), 8192 if n < 10 else 3000) // 4 * 4
    x = 0.1 * torch.randn(n, blocks * N[0], generator=torch.Generator("cuda").manual_seed(n), device="cuda")
    m = PartConvMulti(step_blocks=K)
    m.setup_layout(48000, N[0], n, n, pcs)
    assert m.step_blocks == K
    y = _cut(m, x, [blocks])
    ref = wl.conv_fp64(x[0].cpu().numpy(), pcs[0]["ir"], x.shape[1])
    assert wl.rel_l2(y[0], ref) <= 1e-5
    for sizes in ([12 * K], [44, 4, 12 * K, 4, 100], [16 * K, 4], [28, 12 * K, 60]):
        m.reset()
        assert np.array_equal(_cut(m, x, sizes), y), sizes


@pytest.mark.parametrize("n,N,P,L", [(3, [16, 512], [40, 0], 8000), (5, [64, 256, 4096], [8, 15, 0], 20000),
                                     (24, [32, 1024], [32, 0], 60000)])
def test_mimo_partial_sums_over_several_calls(gpu, n, N, P, L):
    import torch

    rng = np.random.default_rng(L)
    irs = np.stack([wl.decaying_ir(rng, L, 0.3) for _ in range(n * n)]).reshape(n, n, L)
    m = PartConvMIMO()
    m.setup(irs, N, P)
    m.numOutputChannels = n
    blocks = 5 * N[-1] // N[0] + 37
    x = 0.1 * torch.randn(n, blocks * N[0], generator=torch.Generator("cuda").manual_seed(n), device="cuda")
    xs = x.cpu().numpy()
    ref = [sum(wl.conv_fp64(xs[i], irs[i, o], xs.shape[1]) for i in range(n)) for o in range(min(n, 5))]
    for sizes in ([10], [17], [13, 1, 11, 3], [20, 2, 30]):
        m.reset()
        y = _cut(m, x, sizes)
        for o, r in enumerate(ref):
            assert wl.rel_l2(y[o], r) <= 1e-5, (sizes, o)
