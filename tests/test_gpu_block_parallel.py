"""Long calls run block-parallel (csrc/wide.cu), calls of a few blocks and
pc_run one block per launch: the same bits whichever way a signal is cut into
calls, at every block size and part count where the kernels take another
form, and within 1e-5 (relative L2, the parity bound of the other GPU tests)
of the FP64 convolution."""
import numpy as np
import pytest

from partconv_gb300 import PC_INTERLEAVED, PC_PLANAR, PartConvMulti
from partconv_gb300 import workloads as wl
from partconv_gb300.multi import PartConvMultiRelaxed

pytestmark = pytest.mark.gpu

TOL = 1e-5


def _pc(rng, N, P, L, **kw):
    return dict(ir=wl.decaying_ir(rng, L, 0.3), N=N, P=P, **kw)


def _cut(m, x, sizes):
    """x through process() in calls of the given numbers of blocks, the rest in
    one call; a size of 0 stands for one run()."""
    N0, out, at = m.buffer_size, [], 0
    for n in sizes:
        if n == 0:
            y = np.zeros(N0 * m.numOutputChannels, np.float32)
            m.run(y, np.ascontiguousarray(x[at:at + N0]), N0)
            out.append(y.reshape(N0, -1))
            at += N0
        else:
            out.append(m.process(x[at:at + n * N0]))
            at += n * N0
    if at < x.shape[0]:
        out.append(m.process(x[at:]))
    return np.concatenate(out)


# one row per transform size, odd and even powers; part counts 1, 2, 3, one
# more than a tile of 16 and than a register window of 8; level 0 up to 8192
@pytest.mark.parametrize("N,P,L", [
    ([16], [0], 16), ([16], [0], 33), ([16, 32], [2, 0], 32 * 19), ([32, 128], [6, 0], 3000), ([64, 512], [8, 0], 4700),
    ([128, 1024], [14, 0], 9000), ([256, 2048], [8, 0], 30000), ([512, 4096], [14, 0], 40000),
    ([1024, 8192], [8, 0], 60000), ([64, 256, 1024, 16384], [6, 6, 15, 0], 60000), ([2048, 8192], [4, 0], 50000),
    ([4096], [0], 20000), ([8192], [0], 30000), ([128, 32768], [256, 0], 70000), ([256], [0], 256 * 67 + 1)])
def test_any_cut_gives_the_same_bits(gpu, N, P, L):
    rng = np.random.default_rng(L + N[0])
    N0 = N[0]
    blocks = max(40, (L + 2 * N[-1]) // N0 + 9)
    blocks = min(blocks, 1500) + 3
    x = (0.1 * rng.standard_normal((blocks * N0, 1))).astype(np.float32)
    pc = _pc(rng, N, P, L)
    m = PartConvMulti()
    m.setup_layout(48000, N0, 1, 1, [pc])
    y = m.process(x)
    assert wl.rel_l2(y[:, 0], wl.conv_fp64(x[:, 0], pc["ir"], len(x))) <= TOL
    for sizes in ([1, 8, 0, 9, 3], [blocks // 2, 0, 0], [7] * 3 + [blocks // 3, 2, 0]):
        m.reset()
        assert np.array_equal(_cut(m, x, sizes), y), sizes
    m.reset()   # one block per call from the start, then the rest at once
    k = min(70, blocks - 1)
    assert np.array_equal(_cut(m, x, [0] * k), y)


@pytest.mark.parametrize("relaxed", [0, 1])
def test_mixing_layouts_and_cuts(gpu, relaxed):
    rng = np.random.default_rng(5)
    N0 = 64
    pcs = [_pc(rng, [64, 256], [4, 0], 3000, in_ch=0, out_ch=1, scale=0.5), _pc(rng, [64], [0], 900, in_ch=1, out_ch=1),
           _pc(rng, [64, 128], [2, 0], 500, in_ch=1, out_ch=0, mute=1),
           _pc(rng, [64, 512, 4096], [14, 14, 0], 20000, in_ch=2, out_ch=2, scale=-1.0),
           _pc(rng, [64, 512], [8, 0], 5000, in_ch=0, out_ch=1, scale=1.5)]
    x = (0.1 * rng.standard_normal((N0 * 333, 3))).astype(np.float32)
    m = (PartConvMultiRelaxed if relaxed else PartConvMulti)()
    m.setup_layout(48000, N0, 3, 4, pcs)
    y = m.process(x)
    assert not y[:, 0].any() and not y[:, 3].any()
    m.reset()
    assert np.array_equal(m.process(np.ascontiguousarray(x.T), PC_PLANAR).T, y)
    m.reset()
    assert np.array_equal(_cut(m, x, [0, 5, 40, 0, 0, 100, 8]), y)


def test_device_buffers_at_odd_addresses(gpu):
    """Channel rows that start 4 bytes off an 8-byte boundary take the scalar
    loads and stores."""
    import torch

    rng = np.random.default_rng(6)
    N0, frames = 64, 64 * 50
    m = PartConvMulti()
    m.setup_layout(48000, N0, 2, 2, [_pc(rng, [64, 512], [8, 0], 3000, in_ch=c, out_ch=c) for c in range(2)])
    x = torch.randn(2 * frames + 1, device="cuda")
    ys = []
    for off in (0, 1):
        xo = torch.empty(2 * frames + 1, device="cuda")[off:off + 2 * frames].copy_(x[: 2 * frames])
        yo = torch.zeros(2 * frames + 1, device="cuda")[off:off + 2 * frames]
        m.reset()
        m.process_device(yo, xo, frames, PC_PLANAR)
        torch.cuda.synchronize()
        ys.append(yo.cpu().numpy())
    assert np.array_equal(ys[0], ys[1])
    m.reset()
    xi = x[: 2 * frames].view(2, frames).T.contiguous()
    yi = torch.zeros(frames, 2, device="cuda")
    m.process_device(yi, xi, frames, PC_INTERLEAVED)
    torch.cuda.synchronize()
    assert np.array_equal(yi.cpu().numpy().T.ravel(), ys[0])


@pytest.mark.parametrize("K", [2, 4])
@pytest.mark.parametrize("tiles", [None, (64, 4), (512, 64)])
def test_step_blocks_cuts(gpu, K, tiles):
    """Several base blocks per step: short calls (the K-block kernel) and long
    ones give the same bits."""
    rng = np.random.default_rng(7 + K)
    N0 = 64
    pcs = [_pc(rng, [64, 512, 4096], [50, 14, 0], 40000, in_ch=0, out_ch=0), _pc(rng, [64], [0], 130, in_ch=1, out_ch=1),
           _pc(rng, [64, 256], [20, 0], 9000, in_ch=1, out_ch=0)]
    x = (0.1 * rng.standard_normal((N0 * 4 * 90, 2))).astype(np.float32)
    m = PartConvMulti(step_blocks=K, tiles=tiles)
    m.setup_layout(48000, N0, 2, 2, pcs)
    assert m.step_blocks == K
    y = m.process(x)
    for sizes in ([4] * 30, [4, 4, 40, 4, 80]):
        m.reset()
        assert np.array_equal(_cut(m, x, sizes), y), sizes
    ref = sum(wl.conv_fp64(x[:, p["in_ch"]], p["ir"], len(x)) for p in pcs if p["out_ch"] == 0)
    assert wl.rel_l2(y[:, 0], ref) <= TOL
