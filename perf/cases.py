"""Performance cases of the plan API: the transforms that programs run on this provider.

A case is one batched transform executed through a plan:

  kind "c2c"      1D-3D complex transform of `shape` (a text, "64x32"), `batch` of them
  kind "r2c"      real input, numpy.fft.rfftn layout ("c2r": the reverse direction)
  kind "c2r"
  kind "columns"  1D complex transforms down the columns of a row-major [n, batch] matrix, the
                  results stored as rows ("to": "rows"), as columns of a second matrix
                  ("columns"), or rows in and columns out ("from_rows")

with the scalar type, the direction, the normalization and the placement as options. The state a
program holds is the plan and its device buffers; a pass is one execute on the current stream.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(ROOT, "sycl-fft_b200") not in sys.path:
    sys.path.insert(0, os.path.join(ROOT, "sycl-fft_b200"))

import syclfft_b200 as sf  # noqa: E402

MAX_LENGTH = 1 << 20        # longest line of the serving mix
MAX_BYTES = 1 << 27         # input bytes of a drawn smooth transform
MAX_PRIME_BYTES = 1 << 25   # a prime length costs several passes over a longer convolution


def _case(name, kind, shape, batch, scalar, direction, norm, placement="out_of_place", **more):
    return dict(name=name, kind=kind, shape=shape, batch=batch, scalar=scalar, direction=direction, norm=norm,
                placement=placement, **more)


def listed():
    return [
        # one short transform at a time, waiting for each: filters, per-frame spectra (latency)
        _case("single_1024_c64", "c2c", "1024", 1, "float", "forward", "none"),
        # many medium power-of-two lines, the ordinary batched work of signal processing
        _case("batch_4096_c64", "c2c", "4096", 16384, "float", "forward", "orthogonal", "in_place"),
        # a mixed-radix length that fills one SM, inverse direction
        _case("batch_13440_c64", "c2c", "13440", 4096, "float", "backward", "orthogonal", "in_place"),
        # long double-precision lines: more than one SM holds
        _case("batch_65536_c128", "c2c", "65536", 512, "double", "forward", "orthogonal", "in_place"),
        # prime lengths: spectra of records whose length nobody chose
        _case("prime_4099_c128", "c2c", "4099", 256, "double", "forward", "forward"),
        _case("prime_65537_c64", "c2c", "65537", 256, "float", "forward", "forward"),
        # a volume (spectral solvers) and an image in double precision
        _case("cube_256_c64", "c2c", "256x256x256", 1, "float", "backward", "orthogonal", "in_place"),
        _case("plane_2048_c128", "c2c", "2048x2048", 1, "double", "forward", "none"),
        # 7-smooth lengths of a request stream: a line that one block holds, and a longer one
        _case("smooth_3000_c64", "c2c", "3000", 16384, "float", "forward", "none"),
        _case("smooth_680400_c64", "c2c", "680400", 64, "float", "backward", "backward"),
        # real signals, of a length with odd factors
        _case("real_26880_f32", "r2c", "26880", 4096, "float", "forward", "none"),
        # the columns of a row-major matrix, wanted as rows (a corner turn with its transform)
        _case("columns_1024_c64", "columns", "1024", 65536, "float", "forward", "none", to="rows"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def _smooth(rng, lo, hi, even=False):
    """A length without prime factors above 7 in lo..hi, near a log-uniform place."""
    want = _log_int(rng, lo, hi)
    near = []
    p7 = 1
    while p7 <= hi:
        p5 = p7
        while p5 <= hi:
            p3 = p5
            while p3 <= hi:
                p2 = p3
                while p2 <= hi:
                    if p2 >= lo and not (even and p2 % 2):
                        near.append((abs(math.log(p2 / want)), p2))
                    p2 *= 2
                p3 *= 3
            p5 *= 5
        p7 *= 7
    near.sort()
    return rng.choice(near[:8])[1]


def _prime(rng, lo, hi):
    n = _log_int(rng, lo, hi) | 1
    while any(n % d == 0 for d in range(3, math.isqrt(n) + 1, 2)):
        n += 2
    return n if n <= hi else hi


def draw(rng):
    """One more case of the ranges the listed ones stand for."""
    scalar = rng.choice(["float", "float", "float", "double"])
    size = 16 if scalar == "double" else 8
    direction = rng.choice(["forward", "backward"])
    norm = rng.choice(["none", "forward", "backward", "orthogonal"])
    kind = rng.choice(["line", "line", "line", "prime", "grid", "real", "columns"])
    if kind == "line":
        # powers of two and other smooth lengths of the request stream, 1 to many lines
        n = 1 << rng.randint(6, 20) if rng.random() < 0.4 else _smooth(rng, 45, MAX_LENGTH)
        b = _log_int(rng, 1, max(1, min(16384, MAX_BYTES // (n * size))))
        place = rng.choice(["in_place", "out_of_place"])
        norm = "orthogonal" if place == "in_place" else norm
        return _case("line", "c2c", str(n), b, scalar, direction, norm, place)
    if kind == "prime":
        n = _prime(rng, 257, 65537)
        b = _log_int(rng, 1, max(1, min(512, MAX_PRIME_BYTES // (n * size))))
        return _case("prime", "c2c", str(n), b, scalar, direction, norm)
    if kind == "grid":
        rank = rng.choice([2, 3])
        top = 2048 if rank == 2 else 256
        dims = [_smooth(rng, 15, top) for _ in range(rank)]
        b = _log_int(rng, 1, max(1, min(64, MAX_BYTES // (math.prod(dims) * size))))
        place = rng.choice(["in_place", "out_of_place"])
        norm = "orthogonal" if place == "in_place" else norm
        return _case("grid", "c2c", "x".join(map(str, dims)), b, scalar, direction, norm, place)
    if kind == "real":
        n = _smooth(rng, 64, 131072, even=True)
        b = _log_int(rng, 1, max(1, min(16384, MAX_BYTES // (n * size // 2))))
        which = rng.choice(["r2c", "c2r"])
        return _case("real", which, str(n), b, scalar, "forward" if which == "r2c" else "backward", norm)
    n = _smooth(rng, 64, 4096)
    b = _log_int(rng, 16, max(16, min(65536, MAX_BYTES // (n * size))))
    return _case("columns", "columns", str(n), b, scalar, direction, norm, to=rng.choice(["rows", "columns", "from_rows"]))


def _dims(case):
    return [int(v) for v in case["shape"].split("x")]


def _input(case, seed):
    """The input of a case on the GPU: complex [batch, *shape] (or [n, batch] for columns), real
    [batch, n], or the half spectrum of a real signal; uniform in [-1, 1), Gaussian for primes."""
    dims, b, kind = _dims(case), case["batch"], case["kind"]
    real = torch.float64 if case["scalar"] == "double" else torch.float32
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    if kind in ("r2c", "c2r"):
        x = torch.empty([b] + dims, dtype=real, device="cuda").uniform_(-1, 1, generator=g)
        return x if kind == "r2c" else torch.fft.rfft(x.double(), norm="ortho").to(
            torch.complex128 if case["scalar"] == "double" else torch.complex64)
    shape = [dims[0], b] if kind == "columns" and case["to"] != "from_rows" else [b] + dims
    x = torch.empty(shape + [2], dtype=real, device="cuda")
    if len(dims) == 1 and max(dims) > 7 and all(dims[0] % p for p in (2, 3, 5, 7)):
        x.normal_(generator=g)
    else:
        x.uniform_(-1, 1, generator=g)
    return torch.view_as_complex(x)


def prepare(case, seed):
    dims, b, kind = _dims(case), case["batch"], case["kind"]
    x = _input(case, seed)
    options = sf.plan_options(placement=sf.placement[case["placement"]], normalization=sf.normalization[case["norm"]])
    if kind == "r2c":
        plan = sf.plan_dft_r2c_1d(case["scalar"], dims[0], b, options)
        out = torch.empty([b, dims[0] // 2 + 1], dtype=plan.dtype, device="cuda")
    elif kind == "c2r":
        plan = sf.plan_dft_c2r_1d(case["scalar"], dims[0], b, options)
        out = torch.empty([b, dims[0]], dtype=plan.real_dtype, device="cuda")
    elif kind == "columns":
        n = dims[0]
        rows, cols = ((1,), n), ((b,), 1)
        src, dst = {"rows": (cols, rows), "columns": (cols, cols), "from_rows": (rows, cols)}[case["to"]]
        plan = sf.plan_many_dft(case["scalar"], [n], b, sf.direction[case["direction"]], options,
                                layout=sf.data_layout(*src, *dst))
        out = torch.empty([b, n] if case["to"] == "rows" else [n, b], dtype=x.dtype, device="cuda")
    else:
        plan = sf.plan_many_dft(case["scalar"], dims, b, sf.direction[case["direction"]], options)
        out = None if case["placement"] == "in_place" else torch.empty_like(x)
    return dict(plan=plan, x=x, out=out)


def run(state):
    if state["out"] is None:
        state["plan"].execute(state["x"])
        return state["x"]
    state["plan"].execute(state["x"], state["out"])
    return state["out"]


def work(case):
    dims, b, kind = _dims(case), case["batch"], case["kind"]
    size = 16 if case["scalar"] == "double" else 8
    n = math.prod(dims)
    flops = 5.0 * n * math.log2(n) * b
    if kind in ("r2c", "c2r"):
        return {"bytes": b * (n * size // 2 + (n // 2 + 1) * size), "flops": flops / 2}
    return {"bytes": 2 * b * n * size, "flops": flops}


def exact(case, seed):
    dims, kind = _dims(case), case["kind"]
    n = math.prod(dims)
    x = _input(case, seed).cpu().numpy()
    x = x.astype(np.complex128 if np.iscomplexobj(x) else np.float64)
    forward = case["direction"] == "forward"
    # this package scales either direction by 1/n when its normalization names that direction
    scale = {"none": 1.0, "orthogonal": n ** -0.5, "forward": 1.0 / n if forward else 1.0,
             "backward": 1.0 if forward else 1.0 / n}[case["norm"]]
    if kind == "r2c":
        y = np.fft.rfft(x, axis=-1)
    elif kind == "c2r":
        y = np.fft.irfft(x, n=n, axis=-1, norm="forward")
    elif kind == "columns":
        axis = 1 if case["to"] == "from_rows" else 0
        y = np.fft.fft(x, axis=axis) if forward else np.fft.ifft(x, axis=axis, norm="forward")
        y = y if case["to"] == "columns" else np.ascontiguousarray(y.T)
    else:
        axes = tuple(range(1, len(dims) + 1))
        y = np.fft.fftn(x, axes=axes) if forward else np.fft.ifftn(x, axes=axes, norm="forward")
    y *= scale
    return torch.from_numpy(y)
