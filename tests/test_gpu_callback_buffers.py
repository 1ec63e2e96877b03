"""Callbacks use the host block in place or through copies by their size: the bits
of one process() call on either side of each line, with inputs shared by several
PCs, mixed and unused outputs, and the Relaxed class."""
import numpy as np
import pytest

from partconv_gb300 import PartConvMulti
from partconv_gb300 import workloads as wl
from partconv_gb300.multi import PartConvMultiRelaxed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("relaxed", [0, 1])
@pytest.mark.parametrize("N0,n_in,n_out,pcs", [
    (16, 1, 1, 1), (1024, 3, 2, 37), (1024, 3, 2, 38),     # 39936 and 40960 samples over 39 and 40 rows
    (8192, 2, 4, 4), (8192, 2, 4, 5),                      # eight and nine rows
    (64, 40, 40, 300), (64, 33, 3, 700)])                  # below and above with many channels
def test_callback_equals_process(gpu, relaxed, N0, n_in, n_out, pcs):
    rng = np.random.default_rng(N0 + pcs)
    spec = [dict(ir=wl.decaying_ir(rng, 3 * N0 + 7, 0.3), N=[N0], P=[0], in_ch=i * 5 % n_in,
                 out_ch=i % max(1, n_out - 1), scale=1.0 + i % 3, mute=int(i == 3)) for i in range(pcs)]
    m = (PartConvMultiRelaxed if relaxed else PartConvMulti)()
    m.setup_layout(48000, N0, n_in, n_out, spec)
    x = (0.1 * rng.standard_normal((9 * N0, n_in))).astype(np.float32)
    y = np.concatenate([m.process(x[t:t + N0]) for t in range(0, len(x), N0)])
    m.reset()
    out = np.full((9, N0 * n_out), np.nan, np.float32)
    for t in range(9):
        m.run(out[t], np.ascontiguousarray(x[t * N0:(t + 1) * N0]), N0)
    assert np.array_equal(out.reshape(-1, n_out), y)
    n = 9 * N0
    ref = np.zeros((n, n_out))
    for p in spec:
        if not p["mute"]:
            ref[:, p["out_ch"]] += p["scale"] * wl.conv_fp64(x[:, p["in_ch"]], p["ir"], n)
    if relaxed:
        ref = np.concatenate([np.zeros((N0, n_out)), ref[:-N0]])
    assert wl.rel_l2(y, ref) <= 1e-5
