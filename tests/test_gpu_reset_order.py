"""reset() right after calls that are still running on the caller's stream
clears what they leave: the next pass gives a fresh handle's bits."""
import numpy as np
import pytest

from partconv_gb300 import PC_PLANAR, PartConvMulti
from partconv_gb300.mimo import PartConvMIMO

pytestmark = pytest.mark.gpu


def _multi():
    rng = np.random.default_rng(5)
    pcs = [dict(ir=0.05 * rng.standard_normal(40000).astype(np.float32), N=[128, 2048], P=[16, 19], in_ch=i, out_ch=i,
                scale=1.0, mute=0) for i in range(16)]
    m = PartConvMulti()
    m.setup_layout(48000, 128, 16, 16, pcs)
    return m, 16


def _mimo():
    h = 0.05 * np.random.default_rng(6).standard_normal((16, 16, 9000)).astype(np.float32)
    m = PartConvMIMO()
    m.setup(h, [128, 1024], [8, 8])
    return m, 16


@pytest.mark.parametrize("make", [_multi, _mimo])
@pytest.mark.parametrize("steps", [2, 700])
def test_reset_after_running_calls(gpu, make, steps):
    import torch

    frames = 128 * steps
    x = torch.from_numpy((0.1 * np.random.default_rng(7).standard_normal((16, frames))).astype(np.float32)).cuda()
    big = torch.from_numpy((0.1 * np.random.default_rng(8).standard_normal((16, 128 * 3000))).astype(np.float32)).cuda()
    m, _ = make()
    fresh = torch.empty_like(x)
    m.process_device(fresh, x, frames, PC_PLANAR)
    torch.cuda.synchronize()
    y, yb = torch.empty_like(x), torch.empty_like(big)
    for _ in range(3):
        m.process_device(yb, big, big.shape[1], PC_PLANAR)
        m.reset()
        m.process_device(y, x, frames, PC_PLANAR)
        m.reset()
    torch.cuda.synchronize()
    assert torch.equal(y, fresh)
