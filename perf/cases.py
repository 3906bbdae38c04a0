"""The transforms whose speed is measured, each through the public entry points.

A case is a dict of plain values.  ``kind`` names the way it is called:

``c2c``     one complex transform, ``FftPlan.c2c`` + ``execute_checked``
``filter``  forward transform, product with a transfer function, inverse
            transform in place (``execute_in_place``)
``real``    ``FftPlan.r2c`` then ``FftPlan.c2r`` (the spectrum and the signal)
``lines``   ``FftBatch``: lines of mixed lengths in one execute
``front``   ``torch_fft.fftn`` / ``ifftn`` on a tensor

``shape`` is a text ("1920x1080") in the library's order: axis 0 is the
contiguous one.
"""
import functools
import math

import numpy as np
import torch

import wgpufft_b200 as w
from wgpufft_b200 import torch_fft, workloads

_PREC = {"f32": w.FftPrecision.F32, "f64": w.FftPrecision.F64, "df64": w.FftPrecision.Df64}


def listed():
    return [
        # a handful of small images through the torch-shaped front end: a
        # call whose time is its launches and its host path
        {"name": "front_4x64x64", "kind": "front", "shape": "64x64", "batch": 4},
        # short signal frames (a spectrogram block, 4 MiB): one launch, in L2
        {"name": "frames_1024x512", "kind": "c2c", "shape": "1024", "batch": 512,
         "precision": "f32", "inverse": False},
        # frequency-domain filtering of one large image, in place
        {"name": "filter_2048x4096", "kind": "filter", "shape": "2048x4096", "batch": 1},
        # real volume to its spectrum and back (a spectral solver's step)
        {"name": "volume_256", "kind": "real", "shape": "256x256x256", "batch": 1,
         "precision": "f32"},
        # eight full-HD frames, real; sides that are not powers of two
        {"name": "images_1920x1080", "kind": "real", "shape": "1920x1080", "batch": 8,
         "precision": "f32"},
        # awkward lengths, about 256 MiB of lines each: a prime with a smooth
        # p - 1, a prime without one, an odd 13-smooth length
        {"name": "prime_1009", "kind": "c2c", "shape": "1009", "batch": 33255,
         "precision": "f32", "inverse": False},
        {"name": "prime_4099", "kind": "c2c", "shape": "4099", "batch": 8186,
         "precision": "f32", "inverse": False},
        {"name": "smooth_15015", "kind": "c2c", "shape": "15015", "batch": 2234,
         "precision": "f32", "inverse": True},
        # one long line (a whole recording)
        {"name": "line_2e24", "kind": "c2c", "shape": "16777216", "batch": 1,
         "precision": "f32", "inverse": False},
        # the two higher precisions on long lines
        {"name": "f64_2e20x16", "kind": "c2c", "shape": "1048576", "batch": 16,
         "precision": "f64", "inverse": False},
        {"name": "df64_2e20x16", "kind": "c2c", "shape": "1048576", "batch": 16,
         "precision": "df64", "inverse": False},
        # 20,000 lines of mixed lengths in one call (the benchmark's workload)
        {"name": "mixed_20000", "kind": "lines", "lines": 20000, "hi": 65536,
         "lengths_seed": 5, "inverse": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _smooth_near(n):
    """The 13-smooth length nearest to n (the smaller of two)."""
    for d in range(n):
        for m in (n - d, n + d):
            r = m
            for p in (2, 3, 5, 7, 11, 13):
                while r % p == 0:
                    r //= p
            if r == 1:
                return m
    return n


def _side(rng, lo, hi):
    """A side as programs choose them: a power of two, a smooth number, or
    whatever the data has."""
    n = _log_int(rng, lo, hi)
    how = rng.random()
    if how < 1 / 3:
        return 1 << max(1, round(math.log2(n)))
    return _smooth_near(n) if how < 2 / 3 else n


def draw(rng):
    family = rng.choice(["frames", "frames", "long", "nd", "nd", "real", "real", "precise",
                         "lines", "front"])
    inverse = rng.random() < 0.5
    if family == "frames":
        n = _side(rng, 16, 65536)
        points = _log_int(rng, 1 << 19, 1 << 24)
        return {"kind": "c2c", "shape": str(n), "batch": max(1, points // n), "precision": "f32",
                "inverse": inverse}
    if family == "long":
        n = _side(rng, 1 << 17, 1 << 22)
        points = _log_int(rng, 1 << 19, 1 << 23)
        return {"kind": "c2c", "shape": str(n), "batch": max(1, points // n), "precision": "f32",
                "inverse": inverse}
    if family in ("nd", "real"):
        rank = rng.choice([2, 2, 3])
        hi = 2048 if rank == 2 else 200
        shape = [_side(rng, 16, hi) for _ in range(rank)]
        points = _log_int(rng, 1 << 19, 1 << 23)
        batch = max(1, points // math.prod(shape))
        shape = "x".join(map(str, shape))
        if family == "real":
            return {"kind": "real", "shape": shape, "batch": batch,
                    "precision": "f64" if rng.random() < 0.25 else "f32"}
        if rng.random() < 1 / 3:
            return {"kind": "filter", "shape": shape, "batch": batch}
        return {"kind": "c2c", "shape": shape, "batch": batch, "precision": "f32",
                "inverse": inverse}
    if family == "precise":
        n = _side(rng, 64, 1 << 18)
        points = _log_int(rng, 1 << 18, 1 << 21)
        return {"kind": "c2c", "shape": str(n), "batch": max(1, points // n),
                "precision": rng.choice(["f64", "df64"]), "inverse": inverse}
    if family == "lines":
        return {"kind": "lines", "lines": _log_int(rng, 200, 5000),
                "hi": _log_int(rng, 1024, 65536), "lengths_seed": rng.randrange(1 << 30),
                "inverse": inverse}
    return {"kind": "front", "shape": f"{_side(rng, 16, 512)}x{_side(rng, 16, 512)}",
            "batch": _log_int(rng, 1, 32)}


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=4)
def _lengths(lines, hi, seed):
    return workloads.mixed_lengths(lines, seed, 16, hi)


def _case_lengths(case):
    return _lengths(case["lines"], case["hi"], case["lengths_seed"])


def _shape(case):
    return [int(n) for n in case["shape"].split("x")]


def _dims(case):
    return [case["batch"]] + _shape(case)[::-1]


def _normal(case, seed, dims, dtype):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randn(dims, dtype=dtype, device="cuda", generator=g)


def _input(case, seed):
    """The case's input values: iid N(0,1), in the precision it stores."""
    kind = case["kind"]
    if kind == "lines":
        return _normal(case, seed, [int(_case_lengths(case).sum())], torch.complex64)
    if kind == "real":
        dtype = torch.float64 if case["precision"] == "f64" else torch.float32
        return _normal(case, seed, _dims(case), dtype)
    if case.get("precision", "f32") == "f32":
        return _normal(case, seed, _dims(case), torch.complex64)
    return _normal(case, seed, _dims(case), torch.complex128)


def _transfer(case, seed):
    """A filter's transfer function: a smooth low pass with a random phase."""
    phase = _normal(case, seed + 1, _shape(case)[::-1], torch.float32)
    radius = 0.0
    for d in _shape(case)[::-1]:
        f = torch.fft.fftfreq(d, device="cuda")
        radius = (radius[..., None] if torch.is_tensor(radius) else 0.0) + f * f
    return torch.polar(torch.exp(-4.0 * radius), phase)


def _df64_words(z):
    """complex128 as [re_hi, re_lo, im_hi, im_lo] f32 words."""
    v = torch.view_as_real(z)
    hi = v.float()
    lo = (v - hi.double()).float()
    return torch.stack([hi, lo], dim=-1).flatten(-2)


def _config(case, inverse):
    return (w.FftConfig.new_nd(_shape(case)).with_batch(case["batch"])
            .with_direction(w.FftDirection.Inverse if inverse else w.FftDirection.Forward)
            .with_precision(_PREC[case.get("precision", "f32")]))


def prepare(case, seed):
    kind = case["kind"]
    x = _input(case, seed)
    if kind == "front":
        return {"kind": kind, "x": x}
    if kind == "lines":
        lengths = _case_lengths(case)
        direction = w.FftDirection.Inverse if case["inverse"] else w.FftDirection.Forward
        batch = w.FftBatch(lengths, workloads.packed_offsets(lengths), direction=direction,
                           device=0)
        return {"kind": kind, "x": x, "out": torch.empty_like(x), "batch": batch}
    if kind == "c2c":
        if case["precision"] == "df64":
            x = _df64_words(x)
        return {"kind": kind, "x": x, "out": torch.empty_like(x),
                "plan": w.FftPlan.c2c(_config(case, case["inverse"]), device=0)}
    if kind == "filter":
        return {"kind": kind, "x": x, "h": _transfer(case, seed), "work": torch.empty_like(x),
                "forward": w.FftPlan.c2c(_config(case, False), device=0),
                "inverse": w.FftPlan.c2c(_config(case, True), device=0)}
    dims = _dims(case)
    dims[-1] = dims[-1] // 2 + 1
    ctype = torch.complex128 if case["precision"] == "f64" else torch.complex64
    return {"kind": kind, "x": x, "spectrum": torch.empty(dims, dtype=ctype, device="cuda"),
            "signal": torch.empty_like(x),
            "forward": w.FftPlan.r2c(_config(case, False), device=0),
            "inverse": w.FftPlan.c2r(_config(case, True), device=0)}


# -------------------------------------------------------------------- pass
def run(state):
    kind = state["kind"]
    if kind == "c2c":
        state["plan"].execute_checked(state["x"], state["out"])
        return state["out"]
    if kind == "lines":
        state["batch"].execute(state["x"], state["out"])
        return state["out"]
    if kind == "real":
        state["forward"].execute_checked(state["x"], state["spectrum"])
        state["inverse"].execute_checked(state["spectrum"], state["signal"])
        return state["spectrum"], state["signal"]
    if kind == "filter":
        state["forward"].execute_checked(state["x"], state["work"])
        torch.mul(state["work"], state["h"], out=state["work"])
        state["inverse"].execute_in_place(state["work"])
        return state["work"]
    spectrum = torch_fft.fftn(state["x"], dim=(-2, -1))
    return spectrum, torch_fft.ifftn(spectrum, dim=(-2, -1))


# ------------------------------------------------------------------- floor
def _flops(n):
    return 5.0 * n * math.log2(n) if n > 1 else 0.0


def work(case):
    """Each input read once and each output written once; 5 N log2 N (half
    of it for real transforms)."""
    kind = case["kind"]
    if kind == "lines":
        lengths = _case_lengths(case)
        return {"bytes": 16 * int(lengths.sum()), "flops": sum(_flops(int(n)) for n in lengths)}
    n = math.prod(_shape(case))
    points = n * case["batch"]
    flops = case["batch"] * _flops(n)
    if kind == "front":
        return {"bytes": 16 * points + 8 * points, "flops": 2 * flops}
    if kind == "filter":
        return {"bytes": 16 * points + 8 * n, "flops": 2 * flops + 6 * points}
    if kind == "real":
        scalar = 8 if case["precision"] == "f64" else 4
        packed = points // _shape(case)[0] * (_shape(case)[0] // 2 + 1)
        return {"bytes": scalar * (2 * points + 2 * packed), "flops": flops}
    size = 8 if case["precision"] == "f32" else 16
    return {"bytes": 2 * size * points, "flops": flops}


def tolerance(case):
    # About four times the error against 64 bits that the transforms show:
    # f32 0.8e-7 to 3e-7 in the 2-norm (the round trips and Bluestein's
    # convolutions at the upper end), f64 4e-16 to 9e-16, df64 2.3e-13 to
    # 4e-13 (its words are compared as they are; a high word that rounds the
    # other way has a low word that makes up for it).
    precision = case.get("precision", "f32")
    return {"rel": {"f32": 1.2e-6, "f64": 4e-15, "df64": 2e-12}[precision]}


def _fft64(x, inverse, dims):
    return torch.fft.ifftn(x, dim=dims) if inverse else torch.fft.fftn(x, dim=dims)


def exact(case, seed):
    kind = case["kind"]
    x = _input(case, seed)
    dims = list(range(1, 1 + len(_shape(case)))) if kind != "lines" else None
    if kind == "lines":
        host = x.cpu().numpy()
        out = np.empty(host.shape, dtype=np.complex128)
        lengths = _case_lengths(case)
        fft = np.fft.ifft if case["inverse"] else np.fft.fft
        for n, o in zip(lengths, workloads.packed_offsets(lengths)):
            out[o:o + n] = fft(host[o:o + n].astype(np.complex128))
        return torch.from_numpy(out)
    if kind == "front":
        spectrum = torch.fft.fftn(x.to(torch.complex128), dim=(-2, -1))
        return spectrum.cpu(), x.to(torch.complex128).cpu()
    if kind == "real":
        x = x.to(torch.float64)
        order = dims[:-1] + [dims[-1]]
        return torch.fft.rfftn(x, dim=order).cpu(), x.cpu()
    z = x.to(torch.complex128)
    if kind == "filter":
        spectrum = _fft64(z, False, dims) * _transfer(case, seed).to(torch.complex128)
        return _fft64(spectrum, True, dims).cpu()
    if case["precision"] == "df64":
        # the input that the words hold, and the words of the exact result
        v = _df64_words(z).double()
        z = torch.view_as_complex(torch.stack([v[..., 0] + v[..., 1], v[..., 2] + v[..., 3]], -1))
        v = torch.view_as_real(_fft64(z, case["inverse"], dims))
        hi = v.float().double()
        return torch.stack([hi, v - hi], dim=-1).flatten(-2).cpu()
    return _fft64(z, case["inverse"], dims).cpu()
