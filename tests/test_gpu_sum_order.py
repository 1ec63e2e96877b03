"""A decaying response loses nothing of its tail: partial sums over parts run from
the last part to the first.

Input: ones a block apart, so every spectrum, product and transform here is exact
in float32 and only the sum over parts rounds.  Response: 2^24 in the first part
that the partial sums take, then ones four parts apart.  Summed strongest first,
each 1 is half an ulp of 2^24 and is rounded away (3 lost of 3); last to first the
ones meet before they are added to 2^24.  Two roundings at 2^24 are left, half an
ulp (1) each: |y - (2^24 + 3)| <= 2."""
import numpy as np
import pytest

from partconv_gb300 import PartConvMulti

pytestmark = pytest.mark.gpu

BIG = float(1 << 24)


def _outputs(N, P, start, step, at, total, K=1, tiles=None):
    """y at the starts of the steady blocks of `step` samples, by a long call and by
    short ones; the response's parts begin at tap `start`, 2^24 lies in part `at`"""
    ir = np.zeros(start + total * step, np.float32)
    ir[start + at * step] = BIG
    ir[start + (at + 4) * step:start + (at + 13) * step:4 * step] = 1.0
    N0 = N[0]
    frames = (len(ir) // step + 12) * step
    x = np.zeros((frames, 1), np.float32)
    x[::step] = 1.0
    m = PartConvMulti(step_blocks=K, tiles=tiles)
    m.setup_layout(48000, N0, 1, 1, [dict(ir=ir, N=N, P=P)])
    assert m.step_blocks == K
    long = m.process(x)[:, 0]
    m.reset()
    short = np.concatenate([m.process(x[t:t + 4 * N0]) for t in range(0, frames, 4 * N0)])[:, 0]
    first = len(ir) // step
    return long[first * step::step], short[first * step::step]


@pytest.mark.parametrize("N0", [16, 64, 256, 1024, 2048, 4096, 8192, 16384])
@pytest.mark.parametrize("total", [18, 34])
def test_level_0(gpu, N0, total):
    for at in ([2] if total == 18 else [2, 18]):   # the first part of a partial-sum row
        for y in _outputs([N0], [0], 0, N0, at, total):
            assert len(y) >= 8 and np.all(np.abs(y.astype(np.float64) - (BIG + 3)) <= 2), y


@pytest.mark.parametrize("tiles", [(64, 16), (256, 16), (512, 16), (128, 32), (64, 64)])
def test_tuned_tiles(gpu, tiles):
    for y in _outputs([64], [0], 0, 64, 2, 66, tiles=tiles):
        assert np.all(np.abs(y.astype(np.float64) - (BIG + 3)) <= 2), y


@pytest.mark.parametrize("N,P,lo", [([64, 512], [16, 0], 2), ([64, 512], [8, 0], 1), ([64, 128], [2, 0], 1),
                                    ([256, 2048], [16, 0], 2), ([512, 16384], [64, 0], 2)])
def test_larger_levels(gpu, N, P, lo):
    start = N[0] * P[0]
    assert start % N[1] == 0   # the level's blocks begin where the ones lie
    for total in (lo + 16, lo + 17):   # one partial-sum row, and a part over
        for y in _outputs(N, P, start, N[1], lo, total):
            assert np.all(np.abs(y.astype(np.float64) - (BIG + 3)) <= 2), y


@pytest.mark.parametrize("K", [2, 4])
def test_several_blocks_per_step(gpu, K):
    # at most 32 parts are summed one by one; the rows begin somewhere before
    for at in range(32, 48):
        for y in _outputs([64], [0], 0, 64, at, 64, K=K):
            assert np.all(np.abs(y.astype(np.float64) - (BIG + 3)) <= 2), (at, y)
    for y in _outputs([64, 512], [16, 0], 1024, 512, 2, 18, K=K):
        assert np.all(np.abs(y.astype(np.float64) - (BIG + 3)) <= 2), y
