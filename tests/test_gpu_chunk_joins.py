"""Calls longer than one block-parallel chunk: the joins between chunks (ring
wrap, windows that reach back into the chunk before, channel copies of
interleaved input) and pc_process's pieces, whose copies overlap the chunks.
The whole signal has the bits of short calls cut elsewhere and lies within 1e-5
(relative L2) of the float64 convolution."""
import numpy as np
import pytest

from partconv_gb300 import PC_INTERLEAVED, PC_PLANAR, PartConvMulti
from partconv_gb300 import workloads as wl

pytestmark = pytest.mark.gpu

TOL = 1e-5
CHUNK = 4096   # steps of a chunk of a handle this small (the most a chunk takes)


def _handle(rng, N0, n_in, N, L):
    pcs = [dict(ir=wl.decaying_ir(rng, L - 31 * c, 0.3), N=N, P=[8, 64][:len(N) - 1] + [0], in_ch=c, out_ch=c % 2)
           for c in range(n_in)]
    m = PartConvMulti()
    m.setup_layout(48000, N0, n_in, 2, pcs)
    return m, pcs


def _planar(x, layout):
    return x if layout == PC_INTERLEAVED else np.ascontiguousarray(x.T)


def _process(m, x, layout):
    y = m.process(_planar(x, layout), layout)
    return y if layout == PC_INTERLEAVED else y.T


@pytest.mark.parametrize("layout", [PC_INTERLEAVED, PC_PLANAR])
@pytest.mark.parametrize("N0,n_in,N,L,blocks", [
    (16, 2, [16, 128, 1024], 20000, 2 * CHUNK + 808),       # a short last piece
    (16, 5, [16, 64], 700, 2 * CHUNK),                     # copied by channel when interleaved; whole pieces
    (32, 1, [32, 256, 16384], 40000, 3 * CHUNK + 1),       # a last piece of one block; windows longer than a chunk's half
    (64, 1, [64, 512, 32768], 90000, 2 * CHUNK + 17)])     # cluster transforms
def test_pieces_of_a_long_host_call(gpu, layout, N0, n_in, N, L, blocks):
    rng = np.random.default_rng(blocks + n_in)
    m, pcs = _handle(rng, N0, n_in, N, L)
    x = (0.1 * rng.standard_normal((blocks * N0, n_in))).astype(np.float32)

    def launches(k):
        m.reset()
        n = m.kernel_launches()
        _process(m, x[:k * N0], layout)
        return m.kernel_launches() - n

    # a chunk's launches and the one that ends the call: as many chunks as the
    # call's pieces, of 4096 blocks each (the first call also makes the workspace)
    launches(CHUNK)
    full, rest = launches(CHUNK) - 1, launches(blocks % CHUNK) - 1 if blocks % CHUNK > 64 else 0
    n = launches(blocks) - 1
    assert n >= blocks // CHUNK * full + rest and n > full
    m.reset()
    y = _process(m, x, layout)
    for c in range(2):
        ref = sum((wl.conv_fp64(x[:, p["in_ch"]], p["ir"], len(x)) for p in pcs if p["out_ch"] == c), np.zeros(len(x)))
        assert wl.rel_l2(y[:, c], ref) <= TOL
    m.reset()
    out, at = [], 0
    for k in [1, 700, 3000, 390, 6, 3, 1500] + [1111] * 20:   # no call crosses a chunk; joins fall within one
        k = min(k, blocks - at)
        if k > 0:
            out.append(_process(m, x[at * N0:(at + k) * N0], layout))
            at += k
    assert at == blocks and np.array_equal(np.concatenate(out), y)


@pytest.mark.parametrize("layout", [PC_INTERLEAVED, PC_PLANAR])
def test_long_device_call_equals_pieces(gpu, layout):
    import torch

    rng = np.random.default_rng(3)
    N0, blocks = 16, 2 * CHUNK + 300
    m, _ = _handle(rng, N0, 4, [16, 128], 2000)
    x = (0.1 * rng.standard_normal((blocks * N0, 4))).astype(np.float32)
    y = _process(m, x, layout)   # host pieces
    m.reset()
    xd = torch.from_numpy(_planar(x, layout)).cuda()
    yd = torch.empty((blocks * N0, 2) if layout == PC_INTERLEAVED else (2, blocks * N0), device="cuda")
    m.process_device(yd, xd, blocks * N0, layout)
    torch.cuda.synchronize()
    got = yd.cpu().numpy()
    assert np.array_equal(got if layout == PC_INTERLEAVED else got.T, y)
