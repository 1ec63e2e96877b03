"""The block-parallel workspace of a MIMO handle (a second copy of the filter
spectra, rings and sums of a chunk): none for short calls, made and replaced as
calls get longer in mid-signal, left out where the GPU has no room or the stream is
being captured.  A handle that grew gives the bits of one that had the largest
workspace from the start, and both lie within 1e-5 of float64."""
import numpy as np
import pytest

from partconv_gb300 import PC_PLANAR
from partconv_gb300 import workloads as wl
from partconv_gb300.mimo import PartConvMIMO

pytestmark = pytest.mark.gpu


def _irs(rng, n_in, n_out, L):
    return np.stack([wl.decaying_ir(rng, L, 0.3) for _ in range(n_in * n_out)]).reshape(n_in, n_out, L)


def _ref(irs, x):
    return np.stack([sum(wl.conv_fp64(x[i], irs[i, o], x.shape[1]) for i in range(len(x))) for o in range(irs.shape[1])])


def _handle(irs, N, P):
    m = PartConvMIMO()
    m.setup(irs, N, P)
    return m


def _cut(m, x, sizes):
    B, at, out = m.buffer_size, 0, []
    for n in list(sizes) + [x.shape[1]]:
        n = min(n, x.shape[1] // B - at)
        if n > 0:
            out.append(m.process(x[:, at * B:(at + n) * B]))
            at += n
    return np.concatenate(out, axis=1)


@pytest.mark.parametrize("N,P,n_in,n_out,L", [
    ([16], [0], 1, 1, 50), ([16, 64], [4, 0], 3, 3, 700), ([64, 256, 1024], [4, 3, 0], 9, 5, 6001),
    ([128, 2048], [16, 0], 3, 4, 2948), ([4096], [0], 2, 3, 9000), ([256, 1024], [4, 0], 33, 6, 5000)])
def test_growing_in_mid_signal(gpu, N, P, n_in, n_out, L):
    rng = np.random.default_rng(L + n_in)
    irs = _irs(rng, n_in, n_out, L)
    x = (0.1 * rng.standard_normal((n_in, 260 * N[0]))).astype(np.float32)
    ref = _ref(irs, x)
    big = _handle(irs, N, P)
    big.process(x)
    for sizes in ([3, 12, 2, 50, 9, 100], [1] * 20 + [33, 5], [40, 11, 150]):
        m = _handle(irs, N, P)
        held = m.device_bytes()
        big.reset()
        want = _cut(big, x, sizes)
        got = _cut(m, x, sizes)
        assert np.array_equal(got, want), sizes
        assert held < m.device_bytes() <= big.device_bytes()
        for o in range(n_out):
            assert wl.rel_l2(got[o], ref[o]) <= 1e-5, (sizes, o)


def test_short_calls_hold_one_copy_of_the_spectra(gpu):
    rng = np.random.default_rng(1)
    N, P, n, L = [64, 512], [16, 0], 24, 9000
    irs = _irs(rng, n, n, L)
    m = _handle(irs, N, P)
    parts = 16 * 66 + -(-(L - 16 * 64) // 512) * 514
    spectra = 8 * n * n * parts
    held = m.device_bytes()
    assert spectra < held < 1.25 * spectra + (4 << 20)
    x = (0.1 * rng.standard_normal((n, 64 * 64))).astype(np.float32)
    m.process(x[:, :8 * 64])
    assert m.device_bytes() == held
    m.process(x)
    assert m.device_bytes() > held + spectra


def test_first_long_call_while_its_stream_is_captured(gpu):
    import torch

    rng = np.random.default_rng(4)
    irs = _irs(rng, 3, 2, 3000)
    blocks = 40
    x = (0.1 * rng.standard_normal((3, blocks * 64))).astype(np.float32)
    m = _handle(irs, [64, 256], [6, 0])
    xd, yd = torch.from_numpy(x).cuda(), torch.zeros(2, blocks * 64, device="cuda")
    held = m.device_bytes()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        m.process_device(yd, xd, blocks * 64, PC_PLANAR)
    assert m.device_bytes() == held
    g.replay()
    torch.cuda.synchronize()
    ref = _ref(irs, x)
    for o in range(2):
        assert wl.rel_l2(yd[o].cpu().numpy(), ref[o]) <= 1e-5


def test_a_captured_workspace_stays(gpu):
    import torch

    rng = np.random.default_rng(14)
    irs = _irs(rng, 3, 3, 3000)
    blocks = 40
    x = torch.from_numpy((0.1 * rng.standard_normal((3, blocks * 64))).astype(np.float32)).cuda()
    long = x.repeat(1, 10)
    m = _handle(irs, [64, 256], [6, 0])
    y, z = torch.zeros_like(x), torch.zeros_like(long)
    m.process_device(y, x, blocks * 64, PC_PLANAR)
    torch.cuda.synchronize()
    want, held = y.clone(), m.device_bytes()
    m.reset()
    y.zero_()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        m.process_device(y, x, blocks * 64, PC_PLANAR)
    m.reset()
    m.process_device(z, long, 10 * blocks * 64, PC_PLANAR)
    m.reset()
    g.replay()
    torch.cuda.synchronize()
    assert m.device_bytes() == held and torch.equal(y, want)
    ref = _ref(irs, long.cpu().numpy())
    for o in range(3):
        assert wl.rel_l2(z[o].cpu().numpy(), ref[o]) <= 1e-5


@pytest.mark.parametrize("left_mb", [700, 200])
def test_no_room_for_the_workspace(gpu, left_mb):
    """16 x 16 paths of 2^17 taps at 1024-sample blocks: 269 MB of spectra, twice.
    With 700 MB left for the second copy and a chunk a short chunk serves, with 200
    MB one-block steps do; with room again the handle uses it."""
    import torch

    rng = np.random.default_rng(8)
    n, N0, L, blocks = 16, 1024, 1 << 17, 200
    irs = _irs(rng, n, n, L)
    x = torch.from_numpy((0.1 * rng.standard_normal((n, blocks * N0))).astype(np.float32)).cuda()
    a = _handle(irs, [N0], [0])
    warm = torch.empty(n, 4 * N0, device="cuda")
    a.process_device(warm, x[:, :4 * N0].contiguous(), 4 * N0, PC_PLANAR)   # (loads the one-block kernels)
    a.reset()
    y, z = torch.empty_like(x), torch.empty_like(x)
    a.process_device(y, x, blocks * N0, PC_PLANAR)
    torch.cuda.synchronize()
    b = _handle(irs, [N0], [0])
    held = b.device_bytes()
    torch.cuda.empty_cache()
    hold = torch.empty(torch.cuda.mem_get_info()[0] - (left_mb << 20), dtype=torch.uint8, device="cuda")
    try:
        b.process_device(z, x, blocks * N0, PC_PLANAR)
        torch.cuda.synchronize()
        got = b.device_bytes() - held
    finally:
        del hold
        torch.cuda.empty_cache()
    assert (0 < got <= 700 << 20) if left_mb == 700 else got == 0
    err = ((y - z).norm() / y.norm()).item()
    assert err <= 1e-6
    b.reset()
    b.process_device(z, x, blocks * N0, PC_PLANAR)
    torch.cuda.synchronize()
    assert b.device_bytes() == a.device_bytes() and torch.equal(y, z)
