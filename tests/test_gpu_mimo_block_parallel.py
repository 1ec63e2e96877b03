"""MIMO: calls of eight or more base blocks run block-parallel, shorter ones
one block per step.  Both, in any order, against the FP64 convolution (relative
L2 <= 1e-5 per output, the bound of the other MIMO tests) at the edges of the
block-parallel sum: odd outputs (pairs), rows of 18, 34 and 66 bins (tiles of 32
and the two bins after them), 8, 9, 16, 17 and 33 blocks of a level, one part,
one input, and levels that ended mid-block in the call before."""
import numpy as np
import pytest

from partconv_gb300 import PC_INTERLEAVED
from partconv_gb300 import workloads as wl
from partconv_gb300.mimo import PartConvMIMO

pytestmark = pytest.mark.gpu

TOL = 1e-5


def _run(m, x, sizes):
    import torch

    xd = torch.from_numpy(np.ascontiguousarray(x.T)).cuda()   # interleaved
    yd = torch.empty((x.shape[1], m.n_out), dtype=torch.float32, device="cuda")
    at, B = 0, m.buffer_size
    blocks = x.shape[1] // B
    for n in list(sizes) + [blocks]:
        n = min(n, blocks - at)
        if n <= 0:
            break
        m.process_device(yd[at * B:], xd[at * B:], n * B, PC_INTERLEAVED)
        at += n
    torch.cuda.synchronize()
    return yd.cpu().numpy().T


@pytest.mark.parametrize("N,P,n_in,n_out,L,blocks", [
    ([16], [0], 1, 1, 50, 8), ([16, 64], [4, 0], 3, 3, 700, 33), ([32, 256], [8, 0], 2, 5, 2500, 70),
    ([64], [0], 5, 2, 64, 17), ([64, 256, 1024], [4, 3, 0], 9, 5, 6001, 101), ([64, 512], [8, 0], 4, 1, 1500, 9),
    ([128, 2048], [16, 0], 3, 4, 2048 + 900, 80),      # one part of 2048
    ([4096], [0], 2, 3, 9000, 9),                      # one level of large blocks
    ([256, 1024], [4, 0], 67, 6, 5000, 24)])           # more inputs than the sum's lanes and warps divide evenly
def test_calls_of_any_length(gpu, N, P, n_in, n_out, L, blocks):
    rng = np.random.default_rng(L + n_in)
    irs = np.stack([wl.decaying_ir(rng, L, 0.3) for _ in range(n_in * n_out)]).reshape(n_in, n_out, L)
    x = (0.1 * rng.standard_normal((n_in, blocks * N[0]))).astype(np.float32)
    m = PartConvMIMO()
    m.setup(irs, N, P)
    ref = [sum(wl.conv_fp64(x[i], irs[i, o], x.shape[1]) for i in range(n_in)) for o in range(n_out)]
    for sizes in ([], [3, 9, 1, 8], [blocks // 2, 2], [1, 1, 8]):
        m.reset()
        y = _run(m, x, sizes)
        for o in range(n_out):
            assert wl.rel_l2(y[o], ref[o]) <= TOL, (sizes, o)
