"""MIMO calls that run block-parallel for certain (their launches show it): one
input, one output, one level of large blocks, rows of 18 bins alone, and calls of
several chunks, each within 1e-5 (relative L2) of the float64 convolution for the
whole signal."""
import numpy as np
import pytest

from partconv_gb300 import PC_PLANAR
from partconv_gb300 import workloads as wl
from partconv_gb300.mimo import PartConvMIMO

pytestmark = pytest.mark.gpu

TOL = 1e-5


def _run(m, x, sizes):
    """x in calls of the given numbers of blocks, the rest in one; the number of launches of each"""
    B, out, launches, at = m.buffer_size, [], [], 0
    blocks = x.shape[1] // B
    for n in list(sizes) + [blocks]:
        n = min(n, blocks - at)
        if n > 0:
            k = m.kernel_launches()
            out.append(m.process(x[:, at * B:(at + n) * B]))
            launches.append((n, m.kernel_launches() - k))
            at += n
    return np.concatenate(out, axis=1), launches


@pytest.mark.parametrize("N,P,n_in,n_out,L,blocks", [
    ([16], [0], 1, 1, 50, 18),                          # one path, rows of 18 bins
    ([16], [0], 1, 1, 13, 12),                          # one part
    ([64, 512], [8, 0], 4, 1, 1500, 40),                # one output
    ([64, 256], [6, 0], 1, 5, 2100, 40),                # one input
    ([4096], [0], 2, 3, 9000, 20),                      # one level of large blocks
    ([16384], [0], 1, 2, 20000, 11),                    # ... the largest
    ([2048, 8192], [6, 0], 2, 1, 30000, 23),
    ([512, 4096], [16, 0], 20, 3, 9000, 600)])          # chunks of 256 steps
def test_block_parallel_for_certain(gpu, N, P, n_in, n_out, L, blocks):
    rng = np.random.default_rng(L + n_in)
    irs = np.stack([wl.decaying_ir(rng, L, 0.3) for _ in range(n_in * n_out)]).reshape(n_in, n_out, L)
    x = (0.1 * rng.standard_normal((n_in, blocks * N[0]))).astype(np.float32)
    m = PartConvMIMO()
    m.setup(irs, N, P)
    ref = [sum(wl.conv_fp64(x[i], irs[i, o], x.shape[1]) for i in range(n_in)) for o in range(n_out)]
    for sizes in ([], [10, 1], [1, blocks - 1]):
        m.reset()
        y, launches = _run(m, x, sizes)
        for n, k in launches:   # one-block steps launch two or three kernels each
            assert n < 10 or k < 2 * n, (n, k)
        assert max(launches)[0] >= 10
        for o in range(n_out):
            assert wl.rel_l2(y[o], ref[o]) <= TOL, (sizes, o)
        if blocks >= 600 and not sizes:   # three chunks of four kernels, then the state
            assert launches[0][1] >= 12
