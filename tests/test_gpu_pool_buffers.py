"""Host buffers of a serving pool's step that the kernels must not use in place:
one buffer for input and output, overlapping ones, and a buffer that runs from one
registration of host memory into another.  The former give the samples of separate
buffers, over steps in which larger levels fire; the latter is refused.  And
channels that were released, through staged and pinned buffers."""
import numpy as np
import pytest

from partconv_gb300 import PartConvError
from partconv_gb300 import workloads as wl
from partconv_gb300.serving import ServingPool, serving_layout

pytestmark = pytest.mark.gpu


def _pool(irs, N0):
    pool = ServingPool(N0, 64 << 20, len(irs))
    for c, h in enumerate(irs):
        assert pool.admit(h, *serving_layout(len(h), N0)) == c
    return pool


def _steps(pool, bi, bo, x):
    """every block of x [steps][channels][N0] through the buffers (tensors [channels][N0])"""
    y = np.zeros_like(x)
    for t in range(len(x)):
        bi.copy_(_t(x[t]))
        pool.step(bi.data_ptr(), bo.data_ptr(), x.shape[1])
        pool.sync()
        y[t] = bo.numpy()
    return y


def _t(a):
    import torch

    return torch.from_numpy(a)


@pytest.mark.parametrize("N0,L", [(64, 9000), (256, 30000), (1024, 20000)])
def test_shared_and_split_buffers(gpu, N0, L):
    import torch

    rng = np.random.default_rng(N0)
    n = 3
    irs = [wl.decaying_ir(rng, L - 500 * c, 0.4) for c in range(n)]
    x = (0.1 * rng.standard_normal((3 * L // N0 // 2 + 8, n, N0))).astype(np.float32)
    sep = _steps(_pool(irs, N0), torch.zeros(n, N0).pin_memory(), torch.zeros(n, N0).pin_memory(), x)
    for c in range(n):
        assert wl.rel_l2(sep[:, c].ravel(), wl.conv_fp64(x[:, c].ravel(), irs[c], x[:, c].size)) <= 1e-5
    one = torch.zeros(2 * n, N0).pin_memory()
    assert np.array_equal(_steps(_pool(irs, N0), one[:n], one[:n], x), sep)              # in place
    assert np.array_equal(_steps(_pool(irs, N0), one[1:n + 1], one[:n], x), sep)         # a row apart
    assert np.array_equal(_steps(_pool(irs, N0), one[:n], one[n - 1:2 * n - 1], x), sep)
    assert np.array_equal(_steps(_pool(irs, N0), one[:n], one[n:], x), sep)              # touching, not overlapping
    flat = torch.zeros(2 * n * N0 + 2).pin_memory()                                      # rows at odd addresses
    bi, bo = flat[1:1 + n * N0].view(n, N0), flat[2 + n * N0:].view(n, N0)
    assert np.array_equal(_steps(_pool(irs, N0), bi, bo, x), sep)


def test_buffer_across_two_registrations_is_refused(gpu):
    """A copy refuses such a buffer; the kernels must not be given it instead."""
    import torch

    n, N0, page = 4, 1024, 1 << 16
    pool = _pool([wl.decaying_ir(np.random.default_rng(2), 9000, 0.4)] * n, N0)
    raw = np.zeros(5 * page // 4, np.float32)
    base = (raw.ctypes.data + page - 1) // page * page
    rt = torch.cuda.cudart()
    regs = [base, base + page]   # two registrations side by side
    for r in regs:
        assert int(rt.cudaHostRegister(r, page, 0)) == 0
    try:
        at = base + page - 2 * N0 * 4   # two rows in each
        with pytest.raises(PartConvError):
            pool.step(at, torch.zeros(n, N0).pin_memory().data_ptr(), n)
    finally:
        torch.cuda.synchronize()
        for r in regs:
            rt.cudaHostUnregister(r)


@pytest.mark.parametrize("pinned", [True, False])
def test_released_channels_are_silent(gpu, pinned):
    """The highest channel, then every channel released while the host goes on
    stepping all of them: zeros, not the last block again; a channel admitted in
    their place sounds at once."""
    import torch

    rng = np.random.default_rng(9)
    n, N0 = 3, 64
    irs = [wl.decaying_ir(rng, 700, 0.4) for _ in range(n)]
    pool = _pool(irs, N0)
    bi, bo = torch.zeros(n, N0), torch.ones(n, N0)
    if pinned:
        bi, bo = bi.pin_memory(), bo.pin_memory()

    def step():
        bi.copy_(_t((0.1 * rng.standard_normal((n, N0))).astype(np.float32)))
        pool.step(bi.data_ptr(), bo.data_ptr(), n)
        pool.sync()
        return [bool(bo[c].any()) for c in range(n)]

    for _ in range(12):
        assert step() == [True, True, True]
    pool.release(2)
    assert [step() for _ in range(3)] == [[True, True, False]] * 3
    pool.release(0)
    assert [step() for _ in range(3)] == [[False, True, False]] * 3
    pool.release(1)
    assert [step() for _ in range(3)] == [[False, False, False]] * 3
    assert pool.admit(irs[0], *serving_layout(700, N0)) == 0
    assert [step() for _ in range(3)] == [[True, False, False]] * 3


def test_channels_admitted_at_any_step(gpu):
    """The larger levels of channels admitted at different steps fire at different
    steps; a class's launch is left out only where none of them does."""
    import torch

    rng = np.random.default_rng(11)
    N0, L, steps = 64, 30000, 700
    at = [0, 3, 17, 130, 131]   # admission steps; one channel leaves before the last comes
    irs = [wl.decaying_ir(rng, L - 100 * c, 0.4) for c in range(len(at))]
    pool = ServingPool(N0, 64 << 20, len(at))
    n = len(at)
    x = (0.1 * rng.standard_normal((steps, n, N0))).astype(np.float32)
    bi, bo = torch.zeros(n, N0).pin_memory(), torch.zeros(n, N0).pin_memory()
    y = np.zeros_like(x)
    for t in range(steps):
        for c in range(n):
            if at[c] == t:
                assert pool.admit(irs[c], *serving_layout(L - 100 * c, N0)) == c
        if t == 400:
            pool.release(1)
        width = sum(a <= t for a in at)
        bi.copy_(_t(x[t]))
        pool.step(bi.data_ptr(), bo.data_ptr(), width)
        pool.sync()
        y[t, :width] = bo[:width].numpy()
    for c in range(n):
        end = 400 if c == 1 else steps
        ref = wl.conv_fp64(x[at[c]:end, c].ravel(), irs[c], (end - at[c]) * N0)
        assert wl.rel_l2(y[at[c]:end, c].ravel(), ref) <= 1e-5
