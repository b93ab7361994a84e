#!/usr/bin/env python
"""Writes conv_catalog.h: the instantiations of conv_kernel.cuh (Bluestein and Rader passes).

    python gen_conv_catalog.py > out               # the committed catalog again (its lines are the timed choices)
    python gen_conv_catalog.py --candidates > candidates.txt   # up to KEEP layouts of every entry
    python gen_conv_catalog.py chosen.txt > out    # the catalog of the chosen lines, with their times

Lengths: single-block convolutions of 2^a * {1, 3, 5, 7} points in float; in double and for the two
factors of a longer convolution those 7-smooth lengths that no longer length beats in time (complex lines
timed on B200), so a convolution of at least 2L - 2 points pads little and costs no slow length. Layouts come
from the model of gen_smooth_catalog.py; the catalog holds the fastest of them with its time at 96 MB.
Rader passes are made where a prime can need them: a single block of length n when n + 1 is prime, columns
of a power of two.
"""
import sys

from gen_smooth_catalog import CC, KK, best, committed, write_catalog, write_parts

KEEP = 9
FLOAT_FUSED = sorted(f << a for f in (1, 3, 5, 7) for a in range(15) if 64 <= f << a <= 16384)
DOUBLE_FUSED = [64, 72, 80, 84, 90, 96, 100, 108, 112, 120, 128, 140, 144, 150, 160, 168, 180, 192, 196, 210, 224, 256,
                288, 320, 336, 360, 392, 400, 432, 448, 480, 512, 560, 640, 672, 768, 800, 864, 896, 960, 1024, 1080,
                1152, 1200, 1260, 1280, 1344, 1440, 1536, 1600, 1728, 1792, 1920, 2016, 2048, 2160, 2304, 2400, 2560,
                2688, 2880, 3072, 3136, 3360, 3584, 3840, 4096, 4480, 4608, 4800, 5120, 5184, 5376, 5760, 6144, 6272,
                6400, 6720, 7168, 7680, 8192]
SPLIT = [64, 72, 80, 84, 90, 96, 100, 108, 112, 120, 128, 144, 160, 168, 180, 192, 196, 210, 224, 240, 256, 288, 320, 336,
         360, 384, 400, 420, 448, 480, 512, 576, 640, 672, 720, 768, 800, 896, 960, 1024]
FUSED, COLS_FWD, ROWS_CONV, COLS_INV = 0, 1, 2, 3


def prime(n):
    return n > 1 and all(n % d for d in range(2, int(n ** 0.5) + 1))


def entry(dbl, kind, rader, l):
    """A candidate; the timing goes in for COST (0 here)."""
    return "%d, %d, %d, %d, %d, %d, %d, %d, %d, %d, 0, %s" % (dbl, kind, rader, l.n, l.tpl, l.w, l.pads, l.pitch, l.threads,
                                                           l.minb(), ", ".join(map(str, l.rs)))


def work(job):
    dbl, kind, n = job
    return job, best(dbl, CC if kind == COLS_FWD else KK, n, KEEP)


def candidates():
    from multiprocessing import Pool
    jobs = [(0, FUSED, n) for n in FLOAT_FUSED] + [(1, FUSED, n) for n in DOUBLE_FUSED]
    jobs += [(d, k, n) for d in (0, 1) for k in (COLS_FWD, ROWS_CONV) for n in SPLIT]
    with Pool() as pool:
        got = dict(pool.map(work, jobs, chunksize=4))
    for dbl, kind, n in jobs:
        for k in (COLS_FWD, COLS_INV) if kind == COLS_FWD else (kind,):
            for rader in (0, 1):
                if rader and (not prime(n + 1) if k == FUSED else k != ROWS_CONV and n & (n - 1)):
                    continue
                yield [entry(dbl, k, rader, l) for l in got[dbl, kind, n]]


HEAD = """// Written by gen_conv_catalog.py: the Bluestein and Rader pass kernels (conv_kernel.cuh).
//
// X(ID, DOUBLE, KIND, RADER, N, TPL, W, PADS, PITCH, MAXT, MINB, COST, RADICES...)
//   KIND 0 fused single pass (whole lines), 1 forward column pass, 2 row convolution pass, 3 inverse column
//   pass; RADER: gather / bin-0 term / scatter in place of the chirp multiplies; COST time per point
//   of the convolution in 10 fs (timed on B200 at 96 MB); the other columns as in smooth_catalog.h.
#pragma once

"""


def write(rows, out):
    out.write(HEAD)
    write_parts(rows, out, "SFB_CONV", 8)
    out.write("#define SFB_CONV_PARTS 8\n")
    write_catalog(out, "SFB_CONV", 8)


def main():
    arg = sys.argv[1] if len(sys.argv) > 1 else ""
    if arg == "--candidates":
        for rows in candidates():
            print("\n".join(rows))
    elif arg:
        with open(arg) as f:
            write([line.strip() for line in f if line.strip()], sys.stdout)
    else:
        write(committed("conv_catalog.h"), sys.stdout)


if __name__ == "__main__":
    main()
