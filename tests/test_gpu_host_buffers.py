"""A serving pool steps on pinned host buffers of exactly its channels without
copies, on any others through them: the same samples either way, zeros for a
released channel between live ones, and larger levels that fire only in some
steps (their launch is skipped in the others)."""
import numpy as np
import pytest

from partconv_gb300 import workloads as wl
from partconv_gb300.serving import ServingPool, serving_layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N0,L", [(64, 9000), (256, 30000), (1024, 20000)])
def test_pinned_and_pageable_buffers_agree(gpu, N0, L):
    import torch

    rng = np.random.default_rng(N0)
    irs = [wl.decaying_ir(rng, L - 500 * c, 0.4) for c in range(3)]
    steps = 3 * L // N0 // 2 + 8
    x = (0.1 * rng.standard_normal((steps, 3, N0))).astype(np.float32)
    got = []
    for pinned, width in ((True, 3), (False, 3), (True, 4)):   # width 4: a channel the pool does not have
        pool = ServingPool(N0, 64 << 20, 4)
        for c in range(3):
            assert pool.admit(irs[c], *serving_layout(len(irs[c]), N0)) == c
        bi, bo = torch.zeros(width, N0), torch.ones(width, N0)
        if pinned:
            bi, bo = bi.pin_memory(), bo.pin_memory()
        y = np.zeros((steps, 3, N0), np.float32)
        for t in range(steps):
            if t == steps - 5:
                pool.release(1)
            bi[:3] = torch.from_numpy(x[t])
            pool.step(bi.data_ptr(), bo.data_ptr(), width)
            pool.sync()
            y[t] = bo[:3].numpy()
        assert not y[steps - 5:, 1].any()
        got.append(y)
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
    for c in (0, 2):
        ref = wl.conv_fp64(x[:, c].ravel(), irs[c], steps * N0)
        assert wl.rel_l2(got[0][:, c].ravel(), ref) <= 1e-5
