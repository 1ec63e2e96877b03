"""pc_convolve_noalloc runs block-parallel in chunks that the static scratch
array can hold: one chunk, several (a long response leaves little room), a call
of a few blocks and a response that leaves none (one block per launch), at odd
device addresses too, against the FP64 convolution (relative L2 <= 1e-5) and,
where both run the same sums, bit for bit against the allocating engine."""
import ctypes as C

import numpy as np
import pytest

from partconv_gb300 import PC_PLANAR, PartConvMulti
from partconv_gb300 import _native as nat
from partconv_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n0,h_len,blocks", [
    (16, 16, 9), (16, 5000, 700), (64, 64 * 18, 130), (64, 64 * 18 + 1, 131), (512, 48000, 40), (1024, 1024 * 3, 4),
    (1024, 1500, 3),                 # fewer blocks than a block-parallel call has
    (1024, 1_450_000, 640),          # several chunks
    (1024, 2_050_000, 6)])           # no room beside the response's spectra
@pytest.mark.parametrize("off", [0, 1])
def test_chunks(gpu, n0, h_len, blocks, off):
    import torch

    rng = np.random.default_rng(h_len + blocks)
    h = wl.decaying_ir(rng, h_len, 0.4)
    frames = n0 * blocks
    x = (0.1 * rng.standard_normal(frames)).astype(np.float32)
    xd = torch.empty(frames + 1, device="cuda")[off:off + frames].copy_(torch.from_numpy(x))
    hd = torch.from_numpy(h).cuda()
    y = torch.full((frames + 1,), float("nan"), device="cuda")[off:off + frames]
    rc = nat.lib().pc_convolve_noalloc(C.c_void_p(xd.data_ptr()), frames, C.c_void_p(hd.data_ptr()), h_len,
                                       C.c_void_p(y.data_ptr()), n0, C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == nat.PC_OK, nat.lib().pc_last_error(None)
    torch.cuda.synchronize()
    got = y.cpu().numpy()
    assert wl.rel_l2(got, wl.conv_fp64(x, h, frames)) <= 1e-5
    if 4 <= blocks and h_len < 2_000_000:
        m = PartConvMulti()
        m.setup_layout(48000, n0, 1, 1, [dict(ir=h, N=[n0], P=[0])])
        ref = torch.empty(1, frames, device="cuda")
        m.process_device(ref, xd, frames, PC_PLANAR)
        torch.cuda.synchronize()
        assert np.array_equal(ref.cpu().numpy()[0], got)
