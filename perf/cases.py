"""Workloads that a user of partconv_gb300 runs, for timing and comparison.

Each case is one way the framework is used: the real-time callback, a long
host buffer, device buffers of many streams or of a mixing matrix, MIMO,
a differentiable layer, a one-shot convolution without allocation and a
serving pool.  IRs are exponentially decaying noise of unit norm (reverb
tails), inputs are N(0, 0.1^2) noise, both drawn on the GPU from the seed.
"""
import math

import numpy as np
import torch

from partconv_gb300 import PC_INTERLEAVED, PC_PLANAR, PartConvMulti
from partconv_gb300.adjoint import PartitionedConv
from partconv_gb300.mimo import PartConvMIMO
from partconv_gb300.multi import PartConvMultiRelaxed
from partconv_gb300.serving import ServingPool, serving_layout
from partconv_gb300.workloads import chain_layout

FS = 48000


def listed():
    return [
        # one channel strip in an audio callback: a short room response at a
        # 64-sample block, one run() per callback (latency and launches)
        dict(name="callback_short", kind="callback", N0=64, ir=3000, blocks=64, layout="chain4"),
        # a long mono reverb in an audio callback: 2^17 taps,
        # 256x8 | 2048x7 | 16384x7
        dict(name="callback_reverb", kind="callback", N0=256, ir=131072, blocks=192, layout="chain8"),
        # the same reverb over a sound file held in host memory
        dict(name="file_mono", kind="file", N0=256, ir=131072, frames=1 << 18, layout="chain8", relaxed=0, channels=1),
        # a six-level layout from a 64-sample block up to 65536 samples, the
        # Relaxed class, stereo file in host memory
        dict(name="file_ladder", kind="file", N0=64, ir=300001, frames=200000, layout="ladder", relaxed=1, channels=2),
        # 32 independent device-resident streams, IRs of 2^14 .. 2^19 taps
        dict(name="streams_32", kind="streams", N0=256, streams=32, ir_lo=1 << 14, ir_hi=1 << 19, frames=1 << 18,
             step_blocks=1),
        # a mixing desk: 6 inputs, 12 filter paths of ragged lengths with
        # scales and one mute, mixed to stereo, interleaved device buffers of
        # an odd number of blocks
        dict(name="mixer_6x2", kind="mixer", N0=128, n_in=6, n_out=2, ir_lo=5000, ir_hi=90000, blocks=1001),
        # 64 x 64 spatial audio matrix, 2^15 taps, 128x16 | 2048x15
        dict(name="mimo_64x64", kind="mimo", N0=128, n_in=64, n_out=64, ir=1 << 15, blocks=128, layout="chain16"),
        # a small ambisonics decoder: 9 inputs, 5 outputs, short responses
        dict(name="mimo_9x5", kind="mimo", N0=64, n_in=9, n_out=5, ir=6001, blocks=301, layout="chain4"),
        # learning a 2^16-tap response from a batch of 8 signals of 2^18
        # samples: forward and both gradients
        dict(name="learn_8", kind="learn", N=512, ratio=8, ir=1 << 16, batch=8, frames=1 << 18, recompute=0),
        # a short odd-sized response over three ragged signals inside a
        # larger model, spectra recomputed in backward
        dict(name="learn_odd", kind="learn", N=128, ratio=8, ir=4999, batch=3, frames=20011, recompute=1),
        # one-shot convolution with no allocation (a plug-in's device buffers)
        dict(name="oneshot", kind="oneshot", N0=512, ir=48000, frames=1 << 17),
        # a serving pool ticking 64 live channels, one step per block
        dict(name="pool_64", kind="pool", N0=256, channels=64, ir_lo=1 << 12, ir_hi=1 << 14, blocks=48),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["callback", "file", "streams", "mixer", "mimo", "learn", "oneshot", "pool"])
    if kind == "callback":
        return dict(kind=kind, N0=rng.choice([32, 64, 128, 256, 512]), ir=_log(rng, 500, 131072),
                    blocks=rng.randint(16, 192), layout=rng.choice(["chain4", "chain8"]))
    if kind == "file":
        return dict(kind=kind, N0=rng.choice([64, 128, 256, 512]), ir=_log(rng, 2000, 300000),
                    frames=_log(rng, 3000, 1 << 18), layout=rng.choice(["chain4", "chain8", "strict8"]),
                    relaxed=rng.randint(0, 1), channels=rng.randint(1, 3))
    if kind == "streams":
        n = _log(rng, 2, 32)
        return dict(kind=kind, N0=rng.choice([64, 128, 256, 512]), streams=n, ir_lo=_log(rng, 1000, 16384),
                    ir_hi=_log(rng, 20000, 1 << 19), frames=_log(rng, 8000, (1 << 18) if n > 8 else (1 << 19)),
                    step_blocks=rng.choice([1, 1, 1, 2, 4]))
    if kind == "mixer":
        return dict(kind=kind, N0=rng.choice([64, 128, 256]), n_in=rng.randint(1, 8), n_out=rng.randint(1, 4),
                    ir_lo=_log(rng, 1000, 8000), ir_hi=_log(rng, 10000, 100000), blocks=_log(rng, 20, 1200))
    if kind == "mimo":
        N0 = rng.choice([64, 128, 256])
        return dict(kind=kind, N0=N0, n_in=_log(rng, 2, 48), n_out=_log(rng, 2, 48), ir=_log(rng, 1000, 1 << 15),
                    blocks=max(1, _log(rng, 500, 1 << 14) // N0), layout=rng.choice(["chain4", "chain8", "chain16"]))
    if kind == "learn":
        return dict(kind=kind, N=rng.choice([128, 256, 512]), ratio=rng.choice([4, 8]), ir=_log(rng, 1000, 1 << 16),
                    batch=rng.randint(1, 8), frames=_log(rng, 5000, 1 << 18), recompute=rng.randint(0, 1))
    if kind == "oneshot":
        return dict(kind=kind, N0=rng.choice([64, 128, 256, 512, 1024]), ir=_log(rng, 500, 100000),
                    frames=_log(rng, 2000, 1 << 17))
    return dict(kind="pool", N0=rng.choice([64, 128, 256, 1024]), channels=_log(rng, 1, 64),
                ir_lo=_log(rng, 800, 4096), ir_hi=_log(rng, 5000, 1 << 14), blocks=rng.randint(8, 64))


# -- layouts and sizes ----------------------------------------------------------
def _layout(case, ir_len):
    kind = case.get("layout", "strict8")
    if kind == "ladder":      # 64x6 | 256x6 | 1024x6 | 4096x6 | 16384x6 | 65536xP
        return [64, 256, 1024, 4096, 16384, 65536], [6, 6, 6, 6, 6, 0]
    if case["kind"] == "mimo":   # a matrix keeps to moderate blocks
        return chain_layout(ir_len, case["N0"], ratio=int(kind[5:]), max_block=2048 if ir_len >= 16384 else 1024)
    if kind == "strict8":     # the slack the reference demands; larger levels have time to spare
        return chain_layout(ir_len, case["N0"], ratio=8, strict=True)
    return chain_layout(ir_len, case["N0"], ratio=int(kind[5:]))


def _up(n, m):
    return (n + m - 1) // m * m


def _ir_lens(case, n):
    """n IR lengths, log-uniform in [ir_lo, ir_hi], both ends among them."""
    if n == 1:
        return [case["ir_hi"]]
    lo, hi = math.log(case["ir_lo"]), math.log(case["ir_hi"])
    # spread evenly, in a fixed shuffled order
    return [int(round(math.exp(lo + (hi - lo) * ((i * 7) % n if math.gcd(7, n) == 1 else i) / (n - 1)))) for i in range(n)]


def _frames(case):
    k = case["kind"]
    if k == "callback" or k == "mixer" or k == "mimo":
        return case["blocks"] * case["N0"]
    if k == "file" or k == "oneshot":
        return _up(case["frames"], case["N0"])
    if k == "streams":
        return _up(case["frames"], case["N0"] * 4)
    if k == "learn":
        return case["frames"]
    raise KeyError(k)


def _paths(case):
    """(in_ch, out_ch, ir_len, scale, mute) of every filter path."""
    k = case["kind"]
    if k in ("callback", "oneshot"):
        return [(0, 0, case["ir"], 1.0, 0)]
    if k == "file":
        return [(c, c, case["ir"] - 17 * c, 1.0, 0) for c in range(case["channels"])]
    if k == "streams":
        return [(i, i, n, 1.0, 0) for i, n in enumerate(_ir_lens(case, case["streams"]))]
    if k == "mixer":
        n = case["n_in"] * case["n_out"]
        lens = _ir_lens(case, n)
        return [(i // case["n_out"], i % case["n_out"], lens[i], 0.5 + 0.25 * (i % 4), int(n > 2 and i == n - 2))
                for i in range(n)]
    if k == "pool":
        return [(i, i, n, 1.0, 0) for i, n in enumerate(_ir_lens(case, case["channels"]))]
    raise KeyError(k)


# -- inputs, drawn on the GPU from the seed ------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _noise(g, *shape):
    return 0.1 * torch.randn(*shape, generator=g, device="cuda")


def _irs(g, rows, length):
    """rows decaying responses: 60 dB over 0.3 .. 2.5 s, unit norm."""
    t60 = 0.3 + 2.2 * torch.rand(rows, 1, generator=g, device="cuda")
    n = torch.arange(length, device="cuda", dtype=torch.float32)[None, :]
    h = torch.randn(rows, length, generator=g, device="cuda") * torch.exp(-6.91 * n / (t60 * FS))
    return h / h.norm(dim=1, keepdim=True)


def _inputs(case, seed):
    """The case's tensors on the GPU: x and h (a list of rows, or one tensor)."""
    g, k = _gen(seed), case["kind"]
    if k == "mimo":
        h = _irs(g, case["n_in"] * case["n_out"], case["ir"]) / case["n_in"]
        return dict(h=h.view(case["n_in"], case["n_out"], case["ir"]), x=_noise(g, case["n_in"], _frames(case)))
    if k == "learn":
        shape = (case["batch"], _frames(case))
        return dict(h=0.01 * torch.randn(case["ir"], generator=g, device="cuda"), x=_noise(g, *shape),
                    gy=torch.randn(*shape, generator=g, device="cuda") / shape[1])
    if k == "pool":
        h = [_irs(g, 1, p[2])[0] for p in _paths(case)]
        x = torch.zeros(case["channels"], _pool_steps(case) * case["N0"], device="cuda")
        x[:, : case["blocks"] * case["N0"]] = _noise(g, case["channels"], case["blocks"] * case["N0"])
        return dict(h=h, x=x)
    n_in = 1 + max(p[0] for p in _paths(case))
    h = [_irs(g, 1, p[2])[0] for p in _paths(case)]
    return dict(h=h, x=_noise(g, n_in, _frames(case)))


def _pool_steps(case):
    """Blocks of signal, then silence until every response has rung out (a
    stream's tail; the pool's channels are then silent again)."""
    flush = 0
    for p in _paths(case):
        N, P = serving_layout(p[2], case["N0"])
        flush = max(flush, sum(n * q for n, q in zip(N, P)) + 2 * N[-1])
    return case["blocks"] + _up(flush, case["N0"]) // case["N0"]


# -- plans ------------------------------------------------------------------------------
def prepare(case, seed):
    k, d = case["kind"], _inputs(case, seed)
    s = dict(kind=k, case=case)
    if k in ("callback", "file", "streams", "mixer"):
        n_in = d["x"].shape[0]
        paths = _paths(case)
        n_out = 1 + max(p[1] for p in paths)
        pcs = []
        for p, h in zip(paths, d["h"]):
            N, P = _layout(case, p[2])
            pcs.append(dict(ir=h.cpu().numpy(), N=N, P=P, in_ch=p[0], out_ch=p[1], scale=p[3], mute=p[4]))
        cls = PartConvMultiRelaxed if case.get("relaxed") else PartConvMulti
        m = cls(step_blocks=case.get("step_blocks", 1))
        m.setup_layout(FS, case["N0"], n_in, n_out, pcs)
        s["m"] = m
        if k == "callback":
            x = d["x"][0].cpu().numpy()
            s["x"] = [np.ascontiguousarray(x[i:i + m.buffer_size]) for i in range(0, x.size, m.buffer_size)]
            s["y"] = np.empty((len(s["x"]), m.buffer_size), np.float32)
        elif k == "file":
            s["x"] = np.ascontiguousarray(d["x"].T.cpu().numpy())
        elif k == "streams":
            s["x"], s["y"] = d["x"], torch.empty(n_out, _frames(case), device="cuda")
        else:
            s["x"], s["y"] = d["x"].T.contiguous(), torch.empty(_frames(case), n_out, device="cuda")
    elif k == "mimo":
        m = PartConvMIMO()
        m.setup(d["h"].cpu().numpy(), *_layout(case, case["ir"]))
        s.update(m=m, x=d["x"], y=torch.empty(case["n_out"], _frames(case), device="cuda"))
    elif k == "learn":
        N, P = chain_layout(case["ir"], case["N"], ratio=case["ratio"], max_block=4096)
        mod = PartitionedConv(d["h"].cpu().numpy(), N, P, case["batch"], case["frames"],
                              recompute=bool(case["recompute"])).cuda()
        s.update(m=mod, x=d["x"].requires_grad_(True), gy=d["gy"])
    elif k == "oneshot":
        from partconv_gb300 import _native

        s.update(lib=_native.lib(), x=d["x"][0].contiguous(), h=d["h"][0].contiguous(),
                 y=torch.empty(_frames(case), device="cuda"))
    else:
        steps = _pool_steps(case)
        pool = ServingPool(case["N0"], 256 << 20, case["channels"])
        ids = []
        for p, h in zip(_paths(case), d["h"]):
            ids.append(pool.admit(h.cpu().numpy(), *serving_layout(p[2], case["N0"])))
        # staging per block, pinned, [step][channel][N0]
        x = d["x"].view(case["channels"], steps, case["N0"]).permute(1, 0, 2).cpu()
        xin = torch.empty(x.shape).pin_memory()
        xin[:, ids] = x
        s.update(m=pool, ids=ids, x=xin, y=torch.empty(x.shape).pin_memory())
    return s


# -- one pass ----------------------------------------------------------------------------
def run(s):
    k, m = s["kind"], s.get("m")
    if k == "callback":         # the host's audio callback, from a stopped transport
        m.reset()
        n = m.buffer_size
        for x, y in zip(s["x"], s["y"]):
            m.run(y, x, n)
        return s["y"]
    if k == "file":
        m.reset()
        return m.process(s["x"], PC_INTERLEAVED)
    if k in ("streams", "mixer", "mimo"):
        # reset() clears the state on the handle's own stream: the work of an
        # earlier pass has to be over
        torch.cuda.current_stream().synchronize()
        m.reset()
        if k == "mixer":
            m.process_device(s["y"], s["x"], s["x"].shape[0], PC_INTERLEAVED)
        else:
            m.process_device(s["y"], s["x"], s["x"].shape[1], PC_PLANAR)
        return s["y"]
    if k == "learn":
        y = m(s["x"])
        gx, gh = torch.autograd.grad(y, (s["x"], m.h), s["gy"])
        return dict(y=y, gx=gx, gh=gh)
    if k == "oneshot":
        rc = s["lib"].pc_convolve_noalloc(s["x"].data_ptr(), s["x"].numel(), s["h"].data_ptr(), s["h"].numel(),
                                          s["y"].data_ptr(), s["case"]["N0"],
                                          torch.cuda.current_stream().cuda_stream)
        assert rc == 0, rc
        return s["y"]
    for i in range(s["x"].shape[0]):   # a tick of the pool per block period
        m.step(s["x"][i].data_ptr(), s["y"][i].data_ptr(), s["x"].shape[1])
        m.sync()
    return s["y"]


# -- the same outputs in 64 bits ------------------------------------------------------------
def _conv64(x, h, n):
    """First n samples of the convolution of x [.., T] and h [.., L], float64."""
    x, h = x.double(), h.double()
    nf = 1 << (x.shape[-1] + h.shape[-1] - 2).bit_length()
    return torch.fft.irfft(torch.fft.rfft(x, nf) * torch.fft.rfft(h, nf), nf)[..., :n]


def exact(case, seed):
    k, d = case["kind"], _inputs(case, seed)
    x, h = d["x"], d["h"]
    if k == "mimo":
        nf = 1 << (x.shape[1] + case["ir"] - 2).bit_length()
        X = torch.fft.rfft(x.double(), nf)
        return torch.stack([torch.fft.irfft((X * torch.fft.rfft(h[:, o].double(), nf)).sum(0), nf)[: x.shape[1]]
                            for o in range(case["n_out"])])
    if k == "learn":
        T = case["frames"]
        gx = _conv64(d["gy"].flip(-1), h[None], T).flip(-1)
        # dL/dh[j] = sum over signals and t of gy[t] x[t - j]
        gh = _conv64(d["gy"], x.flip(-1), 2 * T - 1).sum(0)[T - 1:T - 1 + case["ir"]]
        gh = torch.cat([gh, gh.new_zeros(case["ir"] - gh.numel())])
        return dict(y=_conv64(x, h[None], T), gx=gx, gh=gh)
    n = x.shape[1]
    if k == "oneshot":
        return _conv64(x[0], h[0], n)
    if k == "pool":
        y = torch.stack([_conv64(x[i], h[i], n) for i in range(case["channels"])])
        return y.view(case["channels"], -1, case["N0"]).permute(1, 0, 2).contiguous()
    paths = _paths(case)
    y = x.new_zeros(1 + max(p[1] for p in paths), n, dtype=torch.float64)
    for p, hp in zip(paths, h):
        if not p[4]:
            y[p[1]] += p[3] * _conv64(x[p[0]], hp, n)
    if case.get("relaxed"):     # one base block later
        y = torch.cat([y.new_zeros(y.shape[0], case["N0"]), y[:, : n - case["N0"]]], dim=1)
    if k == "callback":
        return y[0].view(-1, case["N0"])
    return y if k == "streams" else y.T.contiguous()


# -- what one pass cannot do without ----------------------------------------------------------
def _conv_flops(n, taps):
    """Overlap-save with blocks of about the IR's length: two real FFTs
    (2.5 m log2 m each) and one complex product per bin for m / 2 samples."""
    m = 2 << max(4, (max(1, taps) - 1).bit_length())
    m = min(m, 2 << max(4, (n - 1).bit_length()))
    return n / (m / 2) * (2 * 2.5 * m * math.log2(m) + 6 * (m / 2))


def work(case):
    k = case["kind"]
    if k == "mimo":
        n, i, o, L = _frames(case), case["n_in"], case["n_out"], case["ir"]
        m = 2 << max(4, (min(L, n) - 1).bit_length())
        fl = n / (m / 2) * ((i + o) * 2.5 * m * math.log2(m) + 8 * i * o * (m / 2)) * max(1, L / (m / 2))
        return {"bytes": 4.0 * (n * (i + o) + i * o * L), "flops": fl}
    if k == "learn":
        n, b, L = case["frames"], case["batch"], case["ir"]
        return {"bytes": 4.0 * (4 * n * b + 2 * L), "flops": 3 * b * _conv_flops(n, L)}
    if k == "pool":
        n = _pool_steps(case) * case["N0"]
        lens = [p[2] for p in _paths(case)]
        return {"bytes": 4.0 * (2 * n * len(lens) + sum(lens)), "flops": sum(_conv_flops(n, L) for L in lens)}
    n, paths = _frames(case), _paths(case)
    n_in, n_out = 1 + max(p[0] for p in paths), 1 + max(p[1] for p in paths)
    return {"bytes": 4.0 * (n * (n_in + n_out) + sum(p[2] for p in paths)),
            "flops": sum(_conv_flops(n, p[2]) for p in paths)}
