"""Timing cases of the framework's transforms, through its public entry points.

A case names one plan and one exec of it:

  kind   "grid"    one shape: dims (space-separated sides, last contiguous) x batch
         "uneven"  many transforms of different shapes in one plan, one descriptor
                   each, packed back to back in the order they are drawn
  form   "plain"     FP16 in, FP16 out (scaled by 1 / points of a transform)
         "split"     FP32 in, FP32 out
         "split16"   FP16 in, FP32 out
  dir    "forward" or "inverse"
  api    "ptr"   Plan.exec_ptr on device buffers (the C ABI's mcfftExec)
         "torch" Plan.exec on torch tensors
  data   "uniform"  re, im uniform in [-1, 1)
         "wide"     |z| log-uniform in [1e-3, 1e3], phase uniform
         "waves"    eight plane waves and Gaussian noise (a simulation's field)

prepare() makes the inputs, the output buffer and the plan, as a program that
transforms many inputs of one shape does once; run() is one exec.
"""
import math

import numpy as np
import torch

import mcfft_b200 as mc

FORMS = {
    # form: (precision, flags, FP16 input, FP16 output)
    "plain": (mc.PREC_FP16, mc.FLAG_NONE, True, True),
    "split": (mc.PREC_SPLIT, mc.FLAG_NONE, False, False),
    "split16": (mc.PREC_SPLIT, mc.FLAG_INPUT_F16, True, False),
}


def _grid(name, dims, batch, form, direction="forward", api="ptr", data="uniform"):
    return {"name": name, "kind": "grid", "dims": dims, "batch": batch, "form": form,
            "dir": direction, "api": api, "data": data}


def listed():
    return [
        # The smallest call: one frame of a streaming spectrum, where launch and
        # latency are everything.  Called from torch, as an online pipeline does.
        _grid("1d_1024x8_plain_torch", "1024", 8, "plain", api="torch"),
        # The benchmark's small batch of spectra (C1), both precisions.
        _grid("1d_4096x256_plain", "4096", 256, "plain"),
        _grid("1d_4096x256_split16", "4096", 256, "split16"),
        # Short transforms in an odd number (OFDM symbols, short-time spectra):
        # the inverse direction, a ragged last tile.
        _grid("1d_512x9001_plain_inv", "512", 9001, "plain", "inverse"),
        # The headline: long transforms that need a pair of passes (C2), with
        # FP16 samples in; plain and high precision.
        _grid("1d_1048576x64_plain", "1048576", 64, "plain"),
        _grid("1d_1048576x64_split16", "1048576", 64, "split16"),
        # A length whose four-step factors differ, in an odd batch, FP32.
        _grid("1d_131072x37_split_inv", "131072", 37, "split", "inverse"),
        # Images (C3): forward plain, and wide-range FP32 data.
        _grid("2d_1024x1024x16_plain", "1024 1024", 16, "plain"),
        _grid("2d_1024x1024x16_split", "1024 1024", 16, "split", data="wide"),
        # A volume of a spectral solver (C4): FP32, back from the spectrum; and
        # plain, forward.
        _grid("3d_256x256x256_split_inv", "256 256 256", 1, "split", "inverse", data="waves"),
        _grid("3d_256x256x256_plain", "256 256 256", 1, "plain", data="waves"),
        # Everything at once (C5): 4096 1D transforms of 2^8 .. 2^16 points and 64
        # 2D ones, in one plan and one launch.
        {"name": "uneven_4160_plain", "kind": "uneven", "count1d": 4096, "count2d": 64,
         "lo": 8, "hi": 16, "seed": 4, "form": "plain", "dir": "forward", "api": "ptr",
         "data": "uniform"},
    ]


def draw(rng):
    """One more case: sides are powers of two, the batch is any number, and the
    points of a pass lie between 2^13 and 2^26 (FP32: 2^25), spread over the
    logarithm."""
    form = rng.choice(["plain", "plain", "split", "split16"])
    total = 2.0 ** rng.uniform(13, 26 if form == "plain" else 25)
    direction = rng.choice(["forward", "inverse"])
    shape = rng.choice(["1d", "1d", "2d", "3d", "uneven"])
    if shape == "uneven" and total >= 2.0 ** 18:
        count = max(8, int(total / 2.0 ** 14))
        return {"kind": "uneven", "count1d": count, "count2d": count // 64, "lo": rng.choice([7, 8]),
                "hi": rng.choice([14, 16]), "seed": rng.randrange(1 << 30), "form": form,
                "dir": direction, "api": "ptr", "data": "uniform"}
    lg = int(math.log2(total))
    if shape == "2d":
        sides = [rng.randint(5, min(11, lg - 5))]
        sides.append(rng.randint(5, min(11, lg - sides[0])))
    elif shape == "3d" and lg >= 16:
        sides = [rng.randint(5, min(8, lg - 10))]
        sides.append(rng.randint(5, min(8, lg - 5 - sides[0])))
        sides.append(rng.randint(5, min(8, lg - sides[0] - sides[1])))
    else:
        sides = [rng.randint(6, min(24, lg))]
    batch = max(1, int(total / 2 ** sum(sides)))
    data = "wide" if form != "plain" and rng.random() < 0.5 else "uniform"
    return {"kind": "grid", "dims": " ".join(str(1 << s) for s in sides), "batch": batch,
            "form": form, "dir": direction, "api": rng.choice(["ptr", "ptr", "torch"]), "data": data}


def _shapes(case):
    """The transforms of a case, as (shape, batch) runs that lie back to back."""
    if case["kind"] == "grid":
        return [(tuple(int(v) for v in case["dims"].split()), case["batch"])]
    g = np.random.default_rng(case["seed"])
    e = g.integers(case["lo"], case["hi"] + 1, case["count1d"])
    sides = np.array([128, 256, 512])
    nx, ny = (sides[g.integers(0, 3, case["count2d"])] for _ in range(2))
    return [((1 << int(v),), 1) for v in e] + [((int(a), int(b)), 1) for a, b in zip(nx, ny)]


def _points(case):
    return sum(math.prod(shape) * batch for shape, batch in _shapes(case))


def _input(case, seed):
    """The input as interleaved (re, im) on the GPU, in the form's storage type."""
    n = _points(case)
    dev = torch.device("cuda")
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed) * 7919 + 17)
    if case["data"] == "uniform":
        x = torch.rand((n, 2), generator=g, device=dev) * 2 - 1
    elif case["data"] == "wide":
        mag = 10.0 ** (torch.rand(n, generator=g, device=dev) * 6 - 3)
        ph = torch.rand(n, generator=g, device=dev) * (2 * math.pi)
        x = torch.stack([mag * torch.cos(ph), mag * torch.sin(ph)], -1)
    else:
        dims = [int(v) for v in case["dims"].split()]
        x = torch.randn((n, 2), generator=g, device=dev) * 1e-2
        field = torch.zeros(dims, dtype=torch.complex64, device=dev)
        h = np.random.default_rng(int(seed))
        for _ in range(8):
            wave = torch.full((1,), float(h.uniform(0, 1)), dtype=torch.complex64, device=dev)
            for side in dims:
                k = int(h.integers(-(side // 4), side // 4 + 1))
                ph = torch.arange(side, device=dev, dtype=torch.float64) * (2 * math.pi * k / side)
                wave = wave[..., None] * torch.polar(torch.ones_like(ph), ph).to(torch.complex64)
            field += wave.reshape(dims)
        x += torch.view_as_real(field).reshape(-1, 2).repeat(case["batch"], 1)
    return x.to(torch.float16 if FORMS[case["form"]][2] else torch.float32).contiguous()


def prepare(case, seed):
    precision, flags, _, out16 = FORMS[case["form"]]
    x = _input(case, seed)
    y = torch.empty((_points(case), 2), dtype=torch.float16 if out16 else torch.float32,
                    device="cuda")
    if case["kind"] == "grid":
        (shape, batch), = _shapes(case)
        plan = mc.Plan(shape, batch, precision, flags)
    else:
        descs, off = [], 0
        for shape, batch in _shapes(case):
            descs.append((shape, batch, off, off))
            off += math.prod(shape) * batch
        plan = mc.Plan(descs=descs, precision=precision, flags=flags)
    direction = mc.FORWARD if case["dir"] == "forward" else mc.INVERSE
    state = {"plan": plan, "x": x, "y": y, "dir": direction, "api": case["api"]}
    if case["api"] == "torch":
        state["xc"], state["yc"] = torch.view_as_complex(x), torch.view_as_complex(y)
    return state


def run(state):
    plan, x, y = state["plan"], state["x"], state["y"]
    if state["api"] == "torch":
        plan.exec(state["xc"], state["yc"], state["dir"])
    else:
        plan.exec_ptr(x.data_ptr(), y.data_ptr(), state["dir"],
                      torch.cuda.current_stream().cuda_stream)
    return y


def work(case):
    _, _, in16, out16 = FORMS[case["form"]]
    flops = sum(5.0 * math.prod(s) * math.log2(math.prod(s)) * b for s, b in _shapes(case))
    return {"bytes": float(_points(case) * ((4 if in16 else 8) + (4 if out16 else 8))), "flops": flops}


def exact(case, seed):
    """The transform of the same stored input in 64 bits, scaled as the form is."""
    x = torch.view_as_complex(_input(case, seed).to(torch.float64))
    y = torch.empty_like(x)
    off = 0
    for shape, batch in _shapes(case):
        n = math.prod(shape)
        part = x[off:off + n * batch].reshape((batch,) + shape)
        axes = tuple(range(1, len(shape) + 1))
        if case["dir"] == "forward":
            f = torch.fft.fftn(part, dim=axes)
            f = f / n if case["form"] == "plain" else f
        else:
            f = torch.fft.ifftn(part, dim=axes)
            f = f if case["form"] == "plain" else f * n
        y[off:off + n * batch] = f.reshape(-1)
        off += n * batch
    return torch.view_as_real(y)
