"""Device calls whose output is their input (one-level channels, and a square MIMO
matrix): the samples of separate buffers, in long calls, short ones and the calls
after them."""
import numpy as np
import pytest

from partconv_gb300 import PC_INTERLEAVED, PC_PLANAR, PartConvMulti
from partconv_gb300 import workloads as wl
from partconv_gb300.mimo import PartConvMIMO
from partconv_gb300.multi import PartConvMultiRelaxed

pytestmark = pytest.mark.gpu


def _calls(m, x, n_ch, layout, cuts, in_place):
    """x [frames][channels] through device calls of the given numbers of blocks"""
    import torch

    out, at, B = [], 0, m.buffer_size
    for k in cuts:
        xi = x[at:at + k * B]
        buf = torch.from_numpy(np.ascontiguousarray(xi if layout == PC_INTERLEAVED else xi.T)).cuda()
        y = buf if in_place else torch.empty_like(buf)
        m.process_device(y, buf, k * B, layout)
        torch.cuda.synchronize()
        y = y.cpu().numpy()
        out.append(y if layout == PC_INTERLEAVED else y.T)
        at += k * B
    return np.concatenate(out)


@pytest.mark.parametrize("layout", [PC_INTERLEAVED, PC_PLANAR])
@pytest.mark.parametrize("N0,P,K,relaxed", [(64, 5, 1, 0), (64, 40, 4, 0), (1024, 3, 1, 0), (2048, 20, 1, 0), (8192, 2, 1, 0),
                                            (16384, 1, 1, 0), (256, 9, 1, 1)])
def test_one_level_channels(gpu, layout, N0, P, K, relaxed):
    rng = np.random.default_rng(N0 + P)
    n = 3
    pcs = [dict(ir=wl.decaying_ir(rng, N0 * P - 7 * c, 0.3), N=[N0], P=[0], in_ch=c, out_ch=c) for c in range(n)]
    cuts = [40, 4, 12, 4, 60]
    x = (0.1 * rng.standard_normal((sum(cuts) * N0, n))).astype(np.float32)
    got = []
    for in_place in (False, True):
        m = (PartConvMultiRelaxed if relaxed else PartConvMulti)(step_blocks=K)
        m.setup_layout(48000, N0, n, n, pcs)
        got.append(_calls(m, x, n, layout, cuts, in_place))
    assert np.array_equal(got[0], got[1])


@pytest.mark.parametrize("layout", [PC_INTERLEAVED, PC_PLANAR])
@pytest.mark.parametrize("N,P,L", [([64, 512], [8, 0], 3000), ([2048, 16384], [8, 0], 40000)])
def test_square_matrix(gpu, layout, N, P, L):
    rng = np.random.default_rng(L)
    n = 3
    irs = np.stack([wl.decaying_ir(rng, L, 0.3) for _ in range(n * n)]).reshape(n, n, L)
    cuts = [30, 4, 12]
    x = (0.1 * rng.standard_normal((sum(cuts) * N[0], n))).astype(np.float32)
    m = PartConvMIMO()
    m.setup(irs, N, P)
    y = _calls(m, x, n, layout, cuts, True)
    for o in range(n):
        ref = sum(wl.conv_fp64(x[:, i], irs[i, o], len(x)) for i in range(n))
        assert wl.rel_l2(y[:, o], ref) <= 1e-5
