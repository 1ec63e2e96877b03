"""Interleaved input of many channels goes through a copy by channel: it gives
the bits of the planar call, for channel counts around the tile of 32, calls
after a history, of several chunks and too short for the copy, and the first
block against float64 (relative L2 <= 1e-5)."""
import numpy as np
import pytest

from partconv_gb300 import PC_INTERLEAVED, PC_PLANAR, PartConvMulti
from partconv_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_in", [3, 4, 5, 31, 32, 33, 70])
def test_interleaved_equals_planar(gpu, n_in):
    import torch

    rng = np.random.default_rng(n_in)
    N0, cuts = 64, [1, 5, 40, 700, 1100, 8, 4200 if n_in < 6 else 64]
    frames = N0 * sum(cuts)
    ir = [0.05 * rng.standard_normal(1500 + 7 * i).astype(np.float32) for i in range(n_in)]
    pcs = [dict(ir=ir[i], N=[64, 512], P=[14, 2], in_ch=i, out_ch=i % 3, scale=1.0 + i, mute=0) for i in range(n_in)]
    x = (0.1 * rng.standard_normal((frames, n_in))).astype(np.float32)
    xd = torch.from_numpy(x).cuda()
    got = []
    for layout in (PC_INTERLEAVED, PC_PLANAR):
        m = PartConvMulti()
        m.setup_layout(48000, N0, n_in, 3, pcs)
        parts, at = [], 0
        for k in cuts:
            xi = xd[at:at + k * N0]
            at += k * N0
            if layout == PC_INTERLEAVED:
                y = torch.empty(k * N0, 3, device="cuda")
                m.process_device(y, xi.contiguous(), k * N0, layout)
                parts.append(y)
            else:
                y = torch.empty(3, k * N0, device="cuda")
                m.process_device(y, xi.T.contiguous(), k * N0, layout)
                parts.append(y.T)
        got.append(torch.cat(parts).cpu().numpy())
    assert np.array_equal(got[0].view(np.int32), got[1].view(np.int32))
    n = 8 * N0
    ref = np.zeros((n, 3))
    for i in range(n_in):
        ref[:, i % 3] += (1.0 + i) * wl.conv_fp64(x[:n, i], ir[i], n)
    assert wl.rel_l2(got[0][:n], ref) <= 1e-5
