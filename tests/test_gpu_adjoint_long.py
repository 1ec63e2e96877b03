"""A signal of more than 2^31 samples (rows of spectra past 2^31 elements): forward
and both gradients in windows across the whole signal, against float64 (relative
L2 <= 1e-5)."""
import pytest

pytestmark = pytest.mark.gpu

L, W = 3000, 4000


def _conv64(a, b, n):
    import torch

    nf = 1 << (len(a) + len(b) - 2).bit_length()
    return torch.fft.irfft(torch.fft.rfft(a.double(), nf) * torch.fft.rfft(b.double(), nf), nf)[:n]


def _rel(a, b):
    return ((a.double() - b).norm() / b.norm()).item()


def test_more_than_2_31_samples(gpu):
    import torch

    from partconv_gb300.adjoint import DiffPlan, PartitionedConvFunction

    T = (1 << 31) + 20001
    if torch.cuda.mem_get_info()[0] < 120 << 30:
        pytest.skip("needs 85 GB of device memory")
    plan = DiffPlan([256], [12], L, 1, T)
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(1, T, device="cuda", generator=g).requires_grad_(True)
    h = (0.02 * torch.randn(L, device="cuda", generator=g)).requires_grad_(True)
    y = PartitionedConvFunction.apply(x, h, plan, False)
    starts = [0, 1 << 30, (1 << 31) - 2000, T - W]   # dL/dy is zero elsewhere
    gy = torch.zeros_like(y)
    for s in starts:
        gy[0, s:s + W] = torch.randn(W, device="cuda", generator=g)
    gx, gh = torch.autograd.grad(y, (x, h), gy)
    with torch.no_grad():
        ref = torch.zeros(L, dtype=torch.float64, device="cuda")
        for s in starts:
            lo = max(0, s - L + 1)
            xs = x[0, lo:s + W].double()
            assert _rel(y[0, s:s + W], _conv64(xs, h, s + W - lo)[s - lo:]) <= 1e-5, s
            w = gy[0, s:s + W].double()
            want = _conv64(w.flip(0), h, W + L - 1).flip(0)   # dL/dx[s - L + 1 .. s + W)
            assert _rel(gx[0, lo:s + W], want[lo - (s - L + 1):]) <= 1e-5, s
            xs = torch.cat([xs.new_zeros(L - 1 - (s - lo)), xs])
            ref += torch.stack([(w * xs[L - 1 - j:L - 1 - j + W]).sum() for j in range(L)])
        assert _rel(gh, ref) <= 1e-5
    del x, y, gy, gx
    torch.cuda.empty_cache()
