"""The transforms whose speed this repository keeps an eye on, as a user's program calls them.

Each case is a dict of plain values; its "kind" says which entry points a pass goes through:

  fft       bfly.fft / bfly.ifft over the last dimension of a complex64 tensor
  fft_grad  bfly.fft with its gradient (the conjugate transform)
  real      bfly.rfft with its gradient (R2C forward, weighted C2R backward)
  ragged    one launch over requests of many lengths (Plan.make_ragged)
  fft2      bfly.fft2 / bfly.ifft2 over the last two dimensions
  axis      bfly.fft along the last dimension but one
  layer2d   bfly.rfft2 and bfly.irfft2 with the gradients of both
  stft      bfly.stft with the gradient of its signal
  istft     bfly.istft
  host      Plan.run_many: requests in host memory, copies included

Work is counted as what a pass cannot do without: every input read once, every output written
once, 5 n log2 n operations per complex transform of n points (half that for a real one).
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]
if str(ROOT / "ascend-fft_b200") not in sys.path:
    sys.path.insert(0, str(ROOT / "ascend-fft_b200"))

import bfly  # noqa: E402

# Short-time transforms: frame length and hop of speech and music front ends.
FRAMES = ((256, 64), (400, 160), (512, 128), (1024, 256), (1024, 512), (2048, 512), (4096, 1024))


def listed():
    return [
        # one small transform call inside a larger loop: latency of the call
        {"name": "call", "kind": "fft", "n": 256, "batch": 16, "inverse": False},
        # the spectral-layer group of the application mix, 1024 x (8 * 768) rows
        {"name": "batch", "kind": "fft", "n": 1024, "batch": 6144, "inverse": False},
        # 12-carrier resource blocks of an OFDM uplink (DFT spreading), length 2^4 3 5^2
        {"name": "smooth", "kind": "fft", "n": 1200, "batch": 4096, "inverse": False},
        # a length with a large prime factor (17 * 59), as measured series have
        {"name": "prime", "kind": "fft", "n": 1003, "batch": 8192, "inverse": False},
        # long transforms in training, 2^26 points forward and backward
        {"name": "long_grad", "kind": "fft_grad", "n": 32768, "batch": 2048},
        # real transforms in training: R2C forward, its gradient by C2R
        {"name": "real_grad", "kind": "real", "n": 4096, "batch": 1024},
        # a server's mixed queue: 253 requests of 64..4096 points and the OFDM-like, radar-like
        # and spectral-layer-like groups, one launch
        {"name": "queue", "kind": "ragged", "count": 253, "most": 512, "groups": True, "mix": 7},
        # a stack of square images or range-Doppler maps
        {"name": "images", "kind": "fft2", "ny": 1024, "nx": 1024, "batch": 16, "inverse": False},
        # a Fourier-operator layer: 128 channels of 256 x 256, both directions and both gradients
        {"name": "layer2d", "kind": "layer2d", "ny": 256, "nx": 256, "batch": 128},
        # training on ten-second clips at 16 kHz
        {"name": "stft_grad", "kind": "stft", "n": 1024, "hop": 256, "signals": 32, "length": 160000},
        # resynthesis after spectral enhancement, one-minute clips at 16 kHz
        {"name": "istft", "kind": "istft", "n": 512, "hop": 128, "signals": 8, "length": 960000},
        # the grid of 64..4096 points x 1..1024 rows from pinned host memory and back
        {"name": "host", "kind": "host", "most": 1024, "count": 0, "pinned": True, "mix": 0},
    ]


# ------------------------------------------------------------------ more of the same
def _log(rng, lo, hi):
    """An integer in lo..hi, spread evenly over its logarithm."""
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _smooth(n):
    for p in (2, 3, 5, 7, 11, 13):
        while n % p == 0:
            n //= p
    return n == 1


def _length(rng, lo, hi, fits):
    while True:
        n = _log(rng, lo, hi)
        if fits(n):
            return n


def _batch(rng, n, least, most):
    """Rows of n points, least..most points in all; any number of rows, odd ones among them."""
    return max(1, _log(rng, least, most) // n)


def _draw_call(rng):
    return {"kind": "fft", "n": 1 << rng.randint(5, 12), "batch": _log(rng, 1, 64), "inverse": rng.random() < 0.5}


def _draw_batch(rng):
    n = 1 << rng.randint(6, 14)
    return {"kind": "fft", "n": n, "batch": _batch(rng, n, 1 << 18, 1 << 24), "inverse": rng.random() < 0.5}


def _draw_smooth(rng):
    n = _length(rng, 48, 12288, lambda n: _smooth(n) and n & (n - 1))
    return {"kind": "fft", "n": n, "batch": _batch(rng, n, 1 << 18, 1 << 23), "inverse": rng.random() < 0.5}


def _draw_prime(rng):
    n = _length(rng, 17, 8191, lambda n: not _smooth(n))
    return {"kind": "fft", "n": n, "batch": _batch(rng, n, 1 << 18, 1 << 23), "inverse": rng.random() < 0.5}


def _draw_long(rng):
    n = 1 << rng.randint(13, 16)
    return {"kind": "fft_grad", "n": n, "batch": _batch(rng, n, 1 << 20, 1 << 26)}


def _draw_real(rng):
    if rng.random() < 0.7:
        n = 1 << rng.randint(7, 13)
    else:
        n = 2 * _length(rng, 50, 6000, lambda m: _smooth(m) and m & (m - 1))
    return {"kind": "real", "n": n, "batch": _log(rng, 1, max(1, (1 << 24) // n))}


def _draw_ragged(rng):
    return {"kind": "ragged", "count": _log(rng, 16, 253), "most": _log(rng, 16, 512), "groups": rng.random() < 0.5,
            "mix": rng.randrange(1 << 20)}


def _draw_images(rng):
    if rng.random() < 0.7:
        ny, nx = 1 << rng.randint(6, 11), 1 << rng.randint(6, 12)
        return {"kind": "fft2", "ny": ny, "nx": nx, "batch": _batch(rng, ny * nx, ny * nx, 1 << 24),
                "inverse": rng.random() < 0.5}
    n, inner = 1 << rng.randint(5, 12), _log(rng, 8, 1024)
    return {"kind": "axis", "ny": n, "nx": inner, "batch": _batch(rng, n * inner, n * inner, 1 << 24)}


def _draw_layer(rng):
    ny, nx = 1 << rng.randint(5, 9), 1 << rng.randint(6, 10)
    return {"kind": "layer2d", "ny": ny, "nx": nx, "batch": _batch(rng, ny * nx, 1 << 19, 1 << 23)}


def _draw_stft(rng):
    n, hop = rng.choice(FRAMES)
    signals = _log(rng, 1, 32)
    return {"kind": "stft", "n": n, "hop": hop, "signals": signals, "length": _log(rng, 16000, min(960000, 5120000 // signals))}


def _draw_istft(rng):
    return dict(_draw_stft(rng), kind="istft")


def _draw_host(rng):
    return {"kind": "host", "most": _log(rng, 16, 1024), "count": _log(rng, 4, 40), "pinned": rng.random() < 0.75,
            "mix": rng.randrange(1 << 20)}


def draw(rng):
    return rng.choice((_draw_call, _draw_batch, _draw_smooth, _draw_prime, _draw_long, _draw_real, _draw_ragged, _draw_images,
                       _draw_layer, _draw_stft, _draw_istft, _draw_host))(rng)


# ------------------------------------------------------------------ inputs
def _requests(case):
    """(n, batch) of each request of a ragged or host case."""
    if case["kind"] == "host" and not case["count"]:
        return [(n, b) for n in (64, 128, 256, 512, 1024, 2048, 4096) for b in (1, 4, 16, 64, 256, 1024) if b <= case["most"]]
    rng = np.random.default_rng(case["mix"])
    reqs = []
    for _ in range(case["count"]):
        n = 1 << int(rng.integers(6, 13))
        reqs.append((n, max(1, int(round(2.0 ** rng.uniform(0.0, math.log2(case["most"])))))))
    if case.get("groups"):
        reqs += [(2048, 14 * 100), (512, 4096), (1024, 8 * 768)]
    return reqs


def _frames(case):
    return 1 + case["length"] // case["hop"]


def _complex(gen, *shape):
    return torch.randn(*shape, dtype=torch.complex64, device="cuda", generator=gen)


def _real(gen, *shape):
    return torch.rand(*shape, device="cuda", generator=gen) * 2 - 1


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    s = {"case": case}
    if kind == "fft":
        s["x"] = _complex(gen, case["batch"], case["n"])
    elif kind == "fft_grad":
        s["x"] = _complex(gen, case["batch"], case["n"]).requires_grad_(True)
        s["g"] = _complex(gen, case["batch"], case["n"])
    elif kind == "real":
        s["x"] = _real(gen, case["batch"], case["n"]).requires_grad_(True)
        s["g"] = _complex(gen, case["batch"], case["n"] // 2 + 1)
    elif kind in ("fft2", "axis"):
        s["x"] = _complex(gen, case["batch"], case["ny"], case["nx"])
    elif kind == "layer2d":
        shape = (case["batch"], case["ny"], case["nx"])
        s["x"] = _real(gen, *shape).requires_grad_(True)
        s["X"] = torch.fft.rfft2(_real(gen, *shape)).requires_grad_(True)
        s["gX"] = _complex(gen, *shape[:-1], shape[-1] // 2 + 1)
        s["gy"] = _real(gen, *shape)
    elif kind == "stft":
        s["x"] = _real(gen, case["signals"], case["length"]).requires_grad_(True)
        s["w"] = torch.hann_window(case["n"], device="cuda")
        s["g"] = _complex(gen, case["signals"], _frames(case), case["n"] // 2 + 1).transpose(-1, -2)
    elif kind == "istft":
        s["w"] = torch.hann_window(case["n"], device="cuda")
        spec = torch.stft(_real(gen, case["signals"], case["length"]), case["n"], hop_length=case["hop"], window=s["w"],
                          return_complex=True)
        gain = torch.rand(case["signals"], case["n"] // 2 + 1, 1, device="cuda", generator=gen)
        s["X"] = (spec * gain).transpose(-1, -2).contiguous().transpose(-1, -2)   # the layout a short-time transform returns
    elif kind == "ragged":
        reqs = _requests(case)
        total = sum(n * b for n, b in reqs)
        s["x"], s["y"] = _complex(gen, total), torch.empty(total, dtype=torch.complex64, device="cuda")
        s["ctx"] = bfly.Context()
        if s["ctx"].init(device=torch.cuda.current_device()) != 0:
            raise RuntimeError("bfly.Context.init failed")
        s["plan"] = s["ctx"].make_plan()
        at, work = 0, []
        for n, b in reqs:
            work.append((s["x"].data_ptr() + 8 * at, s["y"].data_ptr() + 8 * at, n, b, -1, 1.0))
            at += n * b
        s["work"] = s["plan"].make_ragged(work)
    elif kind == "host":
        reqs = _requests(case)
        total = sum(n * b for n, b in reqs)
        x = torch.empty(2 * total, pin_memory=case["pinned"])
        x.copy_(torch.randn(2 * total, device="cuda", generator=gen))
        s["x"], s["y"] = x.numpy(), torch.empty(2 * total, pin_memory=case["pinned"]).numpy()
        s["keep"] = (x,)
        s["ctx"] = bfly.Context()
        if s["ctx"].init(device=torch.cuda.current_device()) != 0:
            raise RuntimeError("bfly.Context.init failed")
        s["plan"] = s["ctx"].make_plan()
        at, s["work"] = 0, []
        for n, b in reqs:
            end = at + 2 * n * b
            s["work"].append((s["x"][at:end], s["y"][at:end], n, b))
            at = end
    else:
        raise ValueError(kind)
    return s


# ------------------------------------------------------------------ one pass
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "fft":
        return bfly.ifft(s["x"]) if case["inverse"] else bfly.fft(s["x"])
    if kind == "fft_grad":
        y = bfly.fft(s["x"])
        return y, torch.autograd.grad(y, s["x"], s["g"])[0]
    if kind == "real":
        y = bfly.rfft(s["x"])
        return y, torch.autograd.grad(y, s["x"], s["g"])[0]
    if kind == "fft2":
        return bfly.ifft2(s["x"]) if case["inverse"] else bfly.fft2(s["x"])
    if kind == "axis":
        return bfly.fft(s["x"], dim=-2)
    if kind == "layer2d":
        X = bfly.rfft2(s["x"])
        y = bfly.irfft2(s["X"], s=(case["ny"], case["nx"]))
        return (X, y) + torch.autograd.grad((X, y), (s["x"], s["X"]), (s["gX"], s["gy"]))
    if kind == "stft":
        y = bfly.stft(s["x"], case["n"], hop_length=case["hop"], window=s["w"])
        return y, torch.autograd.grad(y, s["x"], s["g"])[0]
    if kind == "istft":
        return bfly.istft(s["X"], case["n"], hop_length=case["hop"], window=s["w"], length=case["length"])
    if kind == "ragged":
        if s["work"].exec(torch.cuda.current_stream().cuda_stream) != 0:
            raise RuntimeError("ragged exec failed")
        return s["y"]
    if s["plan"].run_many(s["work"]) != 0:
        raise RuntimeError("run_many failed")
    return s["y"]


def work(case):
    kind = case["kind"]
    flops = lambda n, rows: 5.0 * n * math.log2(n) * rows  # noqa: E731
    if kind == "fft":
        return {"bytes": 16 * case["n"] * case["batch"], "flops": flops(case["n"], case["batch"])}
    if kind == "fft_grad":
        return {"bytes": 32 * case["n"] * case["batch"], "flops": 2 * flops(case["n"], case["batch"])}
    if kind == "real":
        n, b = case["n"], case["batch"]
        return {"bytes": 2 * (4 * n + 8 * (n // 2 + 1)) * b, "flops": flops(n, b)}
    if kind == "fft2":
        points = case["ny"] * case["nx"]
        return {"bytes": 16 * points * case["batch"], "flops": flops(points, case["batch"])}
    if kind == "axis":
        return {"bytes": 16 * case["ny"] * case["nx"] * case["batch"], "flops": flops(case["ny"], case["nx"] * case["batch"])}
    if kind == "layer2d":
        ny, nx, b = case["ny"], case["nx"], case["batch"]
        return {"bytes": 4 * (4 * nx + 8 * (nx // 2 + 1)) * ny * b, "flops": 2 * flops(ny * nx, b)}
    if kind in ("stft", "istft"):
        n, frames = case["n"], _frames(case) * case["signals"]
        once = {"bytes": 4 * case["signals"] * case["length"] + 8 * (n // 2 + 1) * frames + 4 * n, "flops": flops(n, frames) / 2}
        return {k: (2 if kind == "stft" else 1) * v for k, v in once.items()}
    reqs = _requests(case)
    return {"bytes": sum(16 * n * b for n, b in reqs), "flops": sum(flops(n, b) for n, b in reqs)}


# ------------------------------------------------------------------ the same in 64 bits
def exact(case, seed):
    s = prepare(case, seed)
    kind = case["kind"]
    wide = lambda t: t.detach().to(torch.complex128 if t.is_complex() else torch.float64)  # noqa: E731
    if kind == "fft":
        return torch.fft.ifft(wide(s["x"])) if case["inverse"] else torch.fft.fft(wide(s["x"]))
    if kind in ("fft_grad", "real"):
        x = wide(s["x"]).requires_grad_(True)
        y = torch.fft.fft(x) if kind == "fft_grad" else torch.fft.rfft(x)
        return y.detach(), torch.autograd.grad(y, x, wide(s["g"]))[0]
    if kind == "fft2":
        return torch.fft.ifft2(wide(s["x"])) if case["inverse"] else torch.fft.fft2(wide(s["x"]))
    if kind == "axis":
        return torch.fft.fft(wide(s["x"]), dim=-2)
    if kind == "layer2d":
        x, F = wide(s["x"]).requires_grad_(True), wide(s["X"]).requires_grad_(True)
        X, y = torch.fft.rfft2(x), torch.fft.irfft2(F, s=(case["ny"], case["nx"]))
        return (X.detach(), y.detach()) + torch.autograd.grad((X, y), (x, F), (wide(s["gX"]), wide(s["gy"])))
    if kind == "stft":
        x = wide(s["x"]).requires_grad_(True)
        y = torch.stft(x, case["n"], hop_length=case["hop"], window=wide(s["w"]), return_complex=True)
        return y.detach(), torch.autograd.grad(y, x, wide(s["g"]))[0]
    if kind == "istft":
        return torch.istft(wide(s["X"]), case["n"], hop_length=case["hop"], window=wide(s["w"]), length=case["length"])
    x = wide(s["x"]) if kind == "ragged" else torch.view_as_complex(torch.from_numpy(s["x"]).cuda().double().reshape(-1, 2))
    y, at = torch.empty_like(x), 0
    for n, b in _requests(case):
        y[at:at + n * b] = torch.fft.fft(x[at:at + n * b].reshape(b, n)).reshape(-1)
        at += n * b
    return y if kind == "ragged" else torch.view_as_real(y).reshape(-1)
