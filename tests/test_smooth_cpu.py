"""Host checks of the size-specialised kernels of the 7-smooth lengths: every catalog entry's geometry, their
additional butterflies, and plans stepped thread by thread through the kernel's index arithmetic (bounds,
shared-memory races, twiddle rows, strides) against numpy's FP64 FFT."""
import os
import re

import numpy as np
import pytest

from conftest import fp64_fft, gaussian_complex, norm_scale, rel_l2
from native_libs import butterfly, describe, narrow_lines, real_pair, smooth_run, smooth_run_line

KK, CC, CK, KC = 0, 1, 2, 3


def catalog(name="smooth_catalog.h"):
    src = open(os.path.join(os.path.dirname(__file__), "..", "sycl-fft_b200", "csrc", name)).read()
    return [tuple(int(v) for v in m.split(",")) for m in re.findall(r"X\(([-0-9, ]+)\)", src)]


@pytest.mark.parametrize("radix", [6, 9, 10, 12, 14])
def test_composite_butterflies(radix):
    x = gaussian_complex(radix, radix, np.complex128)
    assert np.max(np.abs(butterfly(radix, x) - np.fft.fft(x))) < 1e-14 * radix
    assert np.max(np.abs(butterfly(radix, x, double=False) - np.fft.fft(x))) < 2e-6 * radix


@pytest.mark.parametrize("radix", [18, 20, 21, 24, 25, 27, 28, 30, 32])
def test_wide_butterflies(radix):
    x = gaussian_complex(radix, radix, np.complex128)
    assert np.max(np.abs(butterfly(radix, x) - np.fft.fft(x))) < 1e-14 * radix
    assert np.max(np.abs(butterfly(radix, x, double=False) - np.fft.fft(x))) < 2e-6 * radix


def test_catalog_geometry():
    """Ids number the entries; radices multiply to the length; lines fit the block, the registers of an
    SM and its shared memory; the padded row holds the line; mappings with a column side take a power of
    two of lines."""
    entries = catalog()
    assert [e[0] for e in entries] == list(range(len(entries)))
    assert len({(e[1], e[2], e[3], e[4]) for e in entries}) == len(entries)
    for e in entries:
        _, dbl, kind, feat, n, tpl, w, pads, pitch, maxt, minb, *radices = e
        assert np.prod(radices) == n and len(radices) >= 2 and max(radices) <= (16 if dbl else 32), e
        assert (w * tpl + 31) // 32 * 32 == maxt <= 1024 and maxt * minb <= 2048, e
        assert pitch > (n - 1) + ((n - 1) >> pads if pads else 0), e
        assert w * pitch * (16 if dbl else 8) <= 227 * 1024, e
        assert kind == KK or w & (w - 1) == 0, e
        assert feat in (0, {KK: 0, CC: 1}.get(kind, 0)) or (kind == KK and feat in (2, 4)), e


def test_pipelined_catalog_geometry():
    """Even float lines, one per block; copy buffer, work buffer and barrier of MINB blocks fit an SM; every
    entry's length has the plain kernel that misaligned buffers and few lines take."""
    entries = catalog("smooth_piped_catalog.h")
    plain = {(e[3], e[4]) for e in catalog() if e[1] == 0 and e[2] == KK}
    assert sorted(e[0] for e in entries) == list(range(len(entries)))
    assert len({(e[3], e[4]) for e in entries}) == len(entries)
    for e in entries:
        _, dbl, kind, feat, n, tpl, w, pads, pitch, maxt, minb, *radices = e
        assert dbl == 0 and kind == KK and w == 1 and feat in (0, 2) and n % 2 == 0 and (feat, n) in plain, e
        assert np.prod(radices) == n and len(radices) >= 2 and max(radices) <= 32, e
        assert (tpl + 31) // 32 * 32 == maxt <= 1024 and maxt * minb <= 2048, e
        assert pitch > (n - 1) + ((n - 1) >> pads if pads else 0), e
        assert minb * ((n + pitch) * 8 + 16 + 1024) <= 228 * 1024 and (n + pitch) * 8 + 16 <= 227 * 1024, e


def test_convolution_catalog_geometry():
    entries = catalog("conv_catalog.h")
    assert [e[0] for e in entries] == list(range(len(entries)))
    assert len({e[1:5] for e in entries}) == len(entries)
    for e in entries:
        _, dbl, kind, rader, n, tpl, w, pads, pitch, maxt, minb, cost, *radices = e
        assert np.prod(radices) == n and len(radices) >= 2 and max(radices) <= 16, e
        assert (w * tpl + 31) // 32 * 32 == maxt <= 1024 and maxt * minb <= 2048, e
        assert pitch > (n - 1) + ((n - 1) >> pads if pads else 0), e
        assert w * pitch * (16 if dbl else 8) <= 227 * 1024, e
        assert kind in (0, 2) or w & (w - 1) == 0, e


# the shortest and longest lines of each mapping, one with idle threads in a stage, several lines per block
@pytest.mark.parametrize("double", [False, True])
@pytest.mark.parametrize("shape,batch", [([18], 70), ([45], 97), ([105], 25), ([810], 3), ([1029], 2), ([3000], 2),
                                         ([6125], 1), ([16807], 1), ([30000], 1), ([65536], 1), ([36, 40], 2),
                                         ([343, 48], 1), ([15, 20, 18], 2), ([25, 2025], 1)], ids=str)
def test_contiguous_plans_by_thread(shape, batch, double):
    n = int(np.prod(shape))
    x = gaussian_complex(n * batch, n + batch, np.complex128)
    for d, norm, ip in ((-1, 3, False), (1, 2, True)):
        y = smooth_run(x, shape, batch, d, norm, double, ip)
        if y is None:
            pytest.skip("a pass of this plan is not a 7-smooth kernel")
        assert rel_l2(y, fp64_fft(x, shape, batch, d, norm_scale(norm, d, n))) < 1e-13


# radices above 16 in every place: two stages of a line, a column and both passes of a four-step, three stages
@pytest.mark.parametrize("shape,batch", [([324], 7), ([500], 3), ([1024], 5), ([945], 2), ([6000], 2), ([12288], 1),
                                         ([810, 24], 1), ([1024, 20], 1), ([291600], 1)], ids=str)
def test_wide_radices_by_thread(shape, batch):
    n = int(np.prod(shape))
    x = gaussian_complex(n * batch, n + batch, np.complex128)
    for d, norm, ip in ((-1, 3, False), (1, 2, True)):
        y = smooth_run(x, shape, batch, d, norm, False, ip)
        assert rel_l2(y, fp64_fft(x, shape, batch, d, norm_scale(norm, d, n))) < 1e-13


# fused and three-pass Bluestein (the shortest and longest block, the first three-pass lengths), Rader in
# one block and in three passes, a prime axis of a grid
@pytest.mark.parametrize("n,batch,double", [
    ([11], 40, False), ([11], 40, True), ([37], 9, True), ([509], 3, True), ([1009], 2, False), ([4099], 1, False),
    ([4099], 1, True), ([8191], 1, False), ([8209], 1, False), ([3583], 1, True), ([257], 5, False), ([641], 3, True),
    ([12289], 1, True), ([19, 17], 2, False),
], ids=str)
def test_convolutions_by_thread(n, batch, double):
    total = int(np.prod(n))
    x = gaussian_complex(total * batch, total + batch, np.complex128)
    for d, norm, ip in ((-1, 1, False), (1, 2, True)):
        y = smooth_run(x, n, batch, d, norm, double, ip)
        if y is None:
            pytest.skip("a pass of this plan is on the general kernel")
        assert rel_l2(y, fp64_fft(x, n, batch, d, norm_scale(norm, d, total))) < 1e-13


@pytest.mark.parametrize("w_lines", [1, 2, 3])
def test_fewer_lines_per_block(w_lines):
    x = gaussian_complex(100 * 7, 3, np.complex128)
    y = smooth_run(x, [100], 7, -1, w_lines=w_lines)
    assert rel_l2(y, fp64_fft(x, [100], 7, -1)) < 1e-13


STRIDED = [
    # (length, lines, in (line stride, element stride), out)
    (64, 24, (1, 24), (64, 1)), (64, 24, (64, 1), (1, 24)), (60, 7, (1, 9), (1, 11)), (100, 5, (107, 1), (103, 1)),
    (2048, 3, (1, 3), (2050, 1)), (1000, 17, (1001, 1), (1, 17)), (16, 1, (1, 3), (16, 1)), (24, 33, (1, 2), (24, 1)),
    (1500, 9, (1, 9), (1500, 1)),
]


@pytest.mark.parametrize("double", [False, True])
@pytest.mark.parametrize("n,b,src,dst", STRIDED, ids=str)
def test_strided_lines_by_thread(n, b, src, dst, double):
    """Strided one-dimensional plans against the transform of the gathered lines: contiguous or padded
    lines, adjacent columns (of any pitch, overlapping reads included) on either side, partial tiles; no
    element outside the output layout is written."""
    at_in = np.arange(b)[:, None] * src[0] + np.arange(n)[None, :] * src[1]
    at_out = np.arange(b)[:, None] * dst[0] + np.arange(n)[None, :] * dst[1]
    x = gaussian_complex(int(at_in.max()) + 1, n + b, np.complex128)
    out = np.full(int(at_out.max()) + 1, 7 - 3j)
    for d, norm in ((-1, 1), (1, 0)):
        y = smooth_run_line(x, n, b, src + dst, out, d, norm, double)
        ref = (np.fft.fft(x[at_in]) if d < 0 else np.fft.ifft(x[at_in]) * n) * norm_scale(norm, d, n)
        assert rel_l2(y[at_out], ref) < 1e-13
        rest = np.ones(out.size, bool)
        rest[at_out.reshape(-1)] = False
        assert np.all(y[rest] == 7 - 3j)


def test_dispatch():
    """Where a plan takes a 7-smooth kernel: whole lines, strided axes and both passes of a four-step;
    not the generic or tensor-core plans, nor passes with Bluestein tables."""
    def ids(shape, **kw):
        return [p["smooth_id"] >= 0 for p in describe(shape, 4, **kw)["passes"]]

    assert ids([3000]) == [True]
    assert ids([680400]) == [True, True]
    assert ids([840, 1200]) == [True, True]
    assert ids([256, 256], split_bf16=True) == [False, False]
    assert ids([1009]) == [False]


def test_three_pass_split():
    """A split convolution is at least 2L - 2 long and not much longer: the pair of catalog lengths whose
    passes take the least time."""
    for n, dbl in ((40009, False), (65521, True), (8209, True), (300007, False)):
        p = describe([n], 2, double=dbl)["passes"]
        assert [x["kind"] for x in p] == ["bluestein_cols_fwd", "bluestein_rows_conv", "bluestein_cols_inv"]
        assert 2 * n - 2 <= p[0]["n"] * p[1]["n"] < 1.25 * (2 * n - 2)


@pytest.mark.parametrize("n", [1, 6, 15])
def test_real_pairs(n):
    """Bins k and n - k of a real line of 2n points from its half-length spectrum, and back."""
    rng = np.random.default_rng(n)
    x = rng.standard_normal(2 * n)
    z = np.fft.fft(x[0::2] + 1j * x[1::2])
    ref = np.fft.rfft(x)
    for k in range(n // 2 + 1):
        w = np.exp(-1j * np.pi * k / n)
        a, c = real_pair(False, z[k], z[(n - k) % n], w)
        assert abs(a - ref[k]) < 1e-12 and abs(c - ref[n - k]) < 1e-12
        p, q = real_pair(True, ref[k], ref[n - k], w)
        assert abs(p - 2 * z[k]) < 1e-12 and (k == 0 or abs(q - 2 * z[n - k]) < 1e-12)


@pytest.mark.parametrize("w", [2, 4, 8, 16])
def test_narrow_arrays_fill_their_tiles(w):
    """Column tiles wider than the array take lines of several outer indices: every line once, in memory
    order; not at and above the tile's width, for one outer index, other mappings or the four-step's columns."""
    for cols in range(1, 17):
        for outer in (1, 2, 3, 7, 64, 1001):
            got = narrow_lines(CC, 0, w, cols, outer)
            if cols >= w or outer == 1 or w == 2:
                assert got is None
                continue
            assert np.array_equal(got[0] * cols + got[1], np.arange(cols * outer)) and got[1].max() == cols - 1
        for kind, feat in ((CC, 1), (KK, 0), (CK, 0), (KC, 0)):
            assert narrow_lines(kind, feat, w, cols, 3) is None


def test_described_kernels():
    """`kernel` names the family that runs a pass, whatever other families it is planned for besides."""
    def names(shape, **kw):
        return [p["kernel"] for p in describe(shape, 4, **kw)["passes"]]

    assert names([3000]) == ["smooth"] and names([4096]) == ["smooth"] and names([680400]) == ["smooth", "smooth"]
    assert names([13440]) == ["piped"] and names([64]) == ["fixed"] and names([64], double=True) == ["smooth"]
    assert names([15]) == ["lean"] and names([1 << 24]) == ["lean", "lean"] and names([7]) == ["general"]
    assert names([1009]) == ["conv"] and names([65537]) == ["conv"] * 3 and names([1009, 6])[1] == "general"
    assert names([256], split_bf16=True) == ["tensor_core"]


@pytest.mark.parametrize("args,name", [(["gen_smooth_catalog.py"], "smooth_catalog.h"),
                                       (["gen_smooth_catalog.py", "--piped"], "smooth_piped_catalog.h"),
                                       (["gen_conv_catalog.py"], "conv_catalog.h")], ids=lambda v: str(v[-1]))
def test_generators_write_the_committed_catalogs(args, name):
    import subprocess
    import sys
    csrc = os.path.join(os.path.dirname(__file__), "..", "sycl-fft_b200", "csrc")
    out = subprocess.run([sys.executable, "-B"] + args, cwd=csrc, capture_output=True, text=True, check=True).stdout
    assert out == open(os.path.join(csrc, name)).read()
