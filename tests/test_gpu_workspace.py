"""The block-parallel workspace of a handle: none for callbacks and short calls,
made by the first long call for its length, moved to a larger one by a longer call
in mid-signal, and a smaller one or none where the GPU has no room.  Results are
the same bits throughout."""
import numpy as np
import pytest

from partconv_gb300 import PartConvMulti
from partconv_gb300 import workloads as wl
from partconv_gb300.multi import PartConvMultiRelaxed

pytestmark = pytest.mark.gpu


def _setup(pcs, N0, n_in=1, n_out=1, cls=PartConvMulti, **kw):
    m = cls(**kw)
    m.setup_layout(48000, N0, n_in, n_out, pcs)
    return m


def _bytes(m):
    return m.info().device_bytes


@pytest.mark.parametrize("N,P,L", [([64, 256], [8, 0], 6000), ([256, 2048, 16384], [8, 7, 0], 131072),
                                   ([1024, 4096, 16384], [8, 7, 0], 131072), ([4096, 16384], [8, 0], 131072),
                                   ([8192], [0], 41000)])
def test_callbacks_and_short_calls_hold_no_workspace(gpu, N, P, L):
    rng = np.random.default_rng(L)
    N0 = N[0]
    m = _setup([dict(ir=wl.decaying_ir(rng, L, 0.3), N=N, P=P)], N0)
    # filter spectra and spectrum ring 16 bytes a tap each (a level's last block
    # in whole), input ring and output rings at most 4 x 4 bytes of the longest
    # reach, twiddles and tables under 2 MB, small maps
    taps = L + sum(N) + 2 * N[-1]
    own = 2 * 16 * taps + 16 * (L + 4 * N[-1]) + (3 << 20)
    before = _bytes(m)
    assert before <= own, (before, own)
    x = (0.1 * rng.standard_normal((40 * N0, 1))).astype(np.float32)
    y = np.zeros(N0, np.float32)
    for t in range(6):
        m.run(y, np.ascontiguousarray(x[t * N0:(t + 1) * N0]), N0)
    m.process(x[:4 * N0])
    assert _bytes(m) - before <= 8 * 4 * N0     # process()'s own device buffers
    m.process(x[:32 * N0])                      # a chunk of 32 steps, not of thousands
    per_step = (16 + 16 + 16) * N0 * len(N)     # spectra, summed spectra, output rings (rounded up)
    rows = sum(2 * 8 * n * 12 + 8 * (L // n + 2) * n + 16 * n for n in N)
    assert _bytes(m) - before <= 8 * 36 * N0 + 40 * per_step + rows + 16 * (L + 4 * N[-1])


CASES = [
    ([16], [0], 700, 1, {}), ([32, 128], [6, 0], 3000, 1, {}), ([64, 256, 1024, 16384], [6, 6, 15, 0], 60000, 1, {}),
    ([256, 2048], [8, 0], 30000, 1, {}), ([128, 32768], [256, 0], 70000, 1, {}), ([4096], [0], 20000, 1, {}),
    ([64, 512, 4096], [14, 14, 0], 20000, 5, {}), ([64, 512, 4096], [50, 14, 0], 40000, 2, dict(step_blocks=4)),
    ([64, 256], [20, 0], 9000, 2, dict(step_blocks=2, tiles=(64, 4))), ([64, 512], [14, 0], 9000, 2, dict(cls="relaxed"))]


@pytest.mark.parametrize("N,P,L,n_in,kw", CASES)
def test_growing_in_mid_signal(gpu, N, P, L, n_in, kw):
    rng = np.random.default_rng(L + n_in)
    N0 = N[0]
    kw = dict(kw)
    cls = PartConvMultiRelaxed if kw.pop("cls", "") else PartConvMulti
    K = kw.get("step_blocks", 1)
    pcs = [dict(ir=wl.decaying_ir(rng, L - 9 * i, 0.3), N=N, P=P, in_ch=i % n_in, out_ch=i % 2, scale=1.0 + i)
           for i in range(n_in + 1)]
    total = 1500 if N0 <= 64 else 420
    x = (0.1 * rng.standard_normal((total * N0, n_in))).astype(np.float32)
    y = _setup(pcs, N0, n_in, 2, cls, **kw).process(x)   # one call, one workspace
    ref = np.zeros((len(x), 2))
    for p in pcs:
        ref[:, p["out_ch"]] += p["scale"] * wl.conv_fp64(x[:, p["in_ch"]], p["ir"], len(x))
    if cls is PartConvMultiRelaxed:
        ref = np.concatenate([np.zeros((N0, 2)), ref[:-N0]])
    assert wl.rel_l2(y, ref) <= 1e-5
    for cuts in ([4, 4, 12, 4, 48, 100], [40, 8, 44, 200], [4] * 17 + [120, 4, 80]):   # K divides each
        m = _setup(pcs, N0, n_in, 2, cls, **kw)
        held, at, out = [_bytes(m)], 0, []
        for k in cuts + [total]:
            k = min(k, total - at)
            if k == 4 and K == 1:   # four callbacks
                for _ in range(4):
                    o = np.zeros(2 * N0, np.float32)
                    m.run(o, np.ascontiguousarray(x[at * N0:(at + 1) * N0]), N0)
                    out.append(o.reshape(N0, 2))
                    at += 1
            else:
                out.append(m.process(x[at * N0:(at + k) * N0]))
                at += k
            held.append(_bytes(m))
        assert np.array_equal(np.concatenate(out), y), cuts
        assert held == sorted(held) and held[0] < held[-1]
        m.reset()
        assert np.array_equal(m.process(x), y)


def test_first_long_call_while_its_stream_is_captured(gpu):
    """No workspace is made then: the graph holds one-block steps, and running it
    gives the samples of the call."""
    import torch

    rng = np.random.default_rng(4)
    N0, blocks = 128, 48
    pcs = [dict(ir=wl.decaying_ir(rng, 9000, 0.3), N=[128, 1024], P=[14, 0])]
    x = torch.from_numpy((0.1 * rng.standard_normal((blocks * N0, 1))).astype(np.float32)).cuda()
    want = _setup(pcs, N0).process(x.cpu().numpy())
    m = _setup(pcs, N0)
    y = torch.zeros(blocks * N0, 1, device="cuda")
    before = _bytes(m)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        m.process_device(y, x, blocks * N0)
    assert _bytes(m) == before
    g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(y.cpu().numpy(), want)
    m.reset()
    y.zero_()
    m.process_device(y, x, blocks * N0)   # and now with one
    torch.cuda.synchronize()
    assert _bytes(m) > before and np.array_equal(y.cpu().numpy(), want)


def test_a_captured_workspace_stays(gpu):
    """A graph of a block-parallel call holds the workspace's addresses: longer
    calls afterwards run in its chunks, and the graph still gives the call."""
    import torch

    rng = np.random.default_rng(14)
    N0, blocks = 128, 40
    pcs = [dict(ir=wl.decaying_ir(rng, 9000, 0.3), N=[128, 1024], P=[14, 0])]
    x = torch.from_numpy((0.1 * rng.standard_normal((20 * blocks * N0, 1))).astype(np.float32)).cuda()
    m = _setup(pcs, N0)
    y, z = torch.zeros(blocks * N0, 1, device="cuda"), torch.zeros_like(x)
    m.process_device(y, x, blocks * N0)
    torch.cuda.synchronize()
    want, held = y.clone(), _bytes(m)
    m.reset()
    y.zero_()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        m.process_device(y, x, blocks * N0)
    m.reset()
    m.process_device(z, x, len(x))          # twenty times as long
    torch.cuda.synchronize()
    assert _bytes(m) == held and torch.equal(z[:blocks * N0], want)
    m.reset()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want)
    n = _setup(pcs, N0)
    w = torch.zeros_like(x)
    n.process_device(w, x, len(x))
    torch.cuda.synchronize()
    assert _bytes(n) > held and torch.equal(w, z)


@pytest.mark.parametrize("left_mb", [330, 160])
def test_no_room_for_the_workspace(gpu, left_mb):
    """32 streams of 8192-sample blocks: a chunk of 64 steps takes about 420 MB, of
    32 steps half of that.  With 330 MB left on the GPU the short chunk serves, with
    160 MB one-block steps do."""
    import torch

    rng = np.random.default_rng(8)
    N0, n, blocks = 8192, 32, 70
    pcs = [dict(ir=wl.decaying_ir(rng, 9000, 0.3), N=[N0], P=[0], in_ch=i, out_ch=i) for i in range(n)]
    x = torch.from_numpy((0.1 * rng.standard_normal((n, blocks * N0))).astype(np.float32)).cuda()
    y, z = torch.empty_like(x), torch.empty_like(x)
    a = _setup(pcs, N0, n, n)
    a.process_device(y, x, blocks * N0, 1)
    one = _setup(pcs[:1], N0)          # (loads the one-block kernels)
    one.process(np.zeros((2 * N0, 1), np.float32))
    torch.cuda.synchronize()
    b = _setup(pcs, N0, n, n)
    before = _bytes(b)
    torch.cuda.empty_cache()
    hold = torch.empty(torch.cuda.mem_get_info()[0] - (left_mb << 20), dtype=torch.uint8, device="cuda")
    try:
        b.process_device(z, x, blocks * N0, 1)
        torch.cuda.synchronize()
        got = _bytes(b) - before
    finally:
        del hold
        torch.cuda.empty_cache()
    assert 0 < got <= 330 << 20 if left_mb == 330 else got == 0
    assert torch.equal(y, z)
    b.reset()                          # with room again
    b.process_device(z, x, blocks * N0, 1)
    torch.cuda.synchronize()
    assert _bytes(b) - before > got and torch.equal(y, z)
