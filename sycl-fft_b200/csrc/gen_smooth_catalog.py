#!/usr/bin/env python
"""Writes smooth_catalog.h: the instantiations of smooth_kernel.cuh, one per 7-smooth length, precision
and thread mapping; and smooth_piped_catalog.h, their copy-engine-pipelined forms.

    python gen_smooth_catalog.py > out            # the committed catalog again (its lines are the timed choices)
    python gen_smooth_catalog.py --candidates > candidates.txt   # up to KEEP layouts of every entry
    python gen_smooth_catalog.py chosen.txt > out # the catalog of the chosen lines
    python gen_smooth_catalog.py --piped [--candidates | chosen.txt]   # the same of smooth_piped_catalog.h

For every length the generator enumerates the radix sequences of the fewest stages (and one more),
the threads per line, and the shared-memory row layouts, and ranks them under a model of one SM's
cycles per line: issue slots of the butterflies, twiddles and addresses, shared-memory wavefronts from
a bank simulation of every exchange, and the bytes in flight of the blocks that fit an SM. The model's
first choices are within 10% of the fastest on average and up to 2x off for single lengths, so the
committed catalog holds the fastest of 20,000 candidates timed on B200 (128 MB of input each). A
complex length is left out where the power-of-two kernel of fixed_catalog.h was faster (64-point float
lines). The real transforms (FEAT 2 and 4) take the layouts chosen for complex lines, or one with a radix
above 16 where that was faster for them. Radices above 16 (float only; the values
of a double butterfly would take twice the registers) are taken where they timed at least 1.5% below the best layout of radices to 16.
A time is the best of three runs of three launches on 128 MB (column mappings: 1024 columns), every candidate in one
process; the chosen lines are the catalogs themselves, which the generator reads back.

Pipelined candidates: the even float lines above 4096 points, one per block, on the layouts timed for the plain
kernel whose copy buffer fits beside them; those that timed at least 5% below the plain kernel are in the catalog.
"""
import itertools
import math
import os
import re
import sys

KK, CC, CK, KC = 0, 1, 2, 3
RADICES = (2, 3, 4, 5, 6, 7, 8, 9, 10, 12, 14, 15, 16, 18, 20, 21, 24, 25, 27, 28, 30, 32)
# floating-point instructions of one butterfly (adds, multiplies, fused multiply-adds)
FP = {2: 4, 3: 14, 4: 16, 5: 40, 6: 40, 7: 78, 8: 56, 9: 104, 10: 100, 12: 104, 14: 184, 15: 190, 16: 160,
      18: 244, 20: 240, 21: 332, 24: 280, 25: 464, 27: 502, 28: 424, 30: 440, 32: 430}
TW_LOADS = {r: (5 if r > 16 else 4 if r > 8 else 3 if r > 4 else 2 if r > 2 else 1) for r in RADICES}
SMEM = 227 * 1024


def max_values(dbl, kind, n):
    """Complex values a thread may hold: 32 float values (radices above 16) take up to 128 registers."""
    return 16 if dbl else 32


KEEP = 8  # candidates per entry that are timed


def smooth(n):
    for p in (2, 3, 5, 7):
        while n % p == 0:
            n //= p
    return n == 1


def multisets(n, stages, top=32):
    if stages == 1:
        return [(n,)] if n in RADICES and n <= top else []
    out = []
    for r in RADICES:
        if r <= top and n % r == 0:
            out += [(r,) + m for m in multisets(n // r, stages - 1, r)]
    return out


def regs(values, dbl):
    """Registers a thread needs for `values` complex values (observed, without spills)."""
    if dbl:
        return 64 if values <= 8 else 76 if values <= 10 else 92 if values <= 12 else 120
    return 40 if values <= 8 else 48 if values <= 10 else 56 if values <= 16 else 72 if values <= 20 else 96 if values <= 25 else 112 if values <= 28 else 128


def conflicts(addr, per):
    """Wavefronts of one warp access: element addresses of the active lanes, `per` lanes at a time."""
    waves = 0
    for h in range(0, len(addr), per):
        banks = {}
        for a in addr[h:h + per]:
            if a is not None:
                banks.setdefault(a % per, set()).add(a)
        if banks:
            waves += max(len(v) for v in banks.values())
    return waves


class Layout:
    def __init__(self, dbl, kind, n, rs, tpl, w, pads, pitch):
        self.dbl, self.kind, self.n, self.rs, self.tpl, self.w, self.pads, self.pitch = dbl, kind, n, rs, tpl, w, pads, pitch
        self.threads = (w * tpl + 31) // 32 * 32

    def lane(self, tid, cmap):
        return (tid % self.w, tid // self.w) if cmap else (tid // self.tpl, tid % self.tpl)

    def at(self, w, k):
        return w * self.pitch + (k + (k >> self.pads) if self.pads else k)

    def waves(self):
        """Shared-memory wavefronts per tile of each stage (a sample of warps, scaled up)."""
        per = 8 if self.dbl else 16
        warps = self.threads // 32
        sample = sorted(set([0, warps // 2, max(0, warps - 2)]))
        out, ns = [], 1
        for s, r in enumerate(self.rs):
            first, last = s == 0, s == len(self.rs) - 1
            cmap = self.kind == CC or (self.kind == CK and first) or (self.kind == KC and last)
            nr = self.n // r
            nb = -(-nr // self.tpl)
            total = 0.0
            for store in (False, True):
                if (first and not store) or (last and store):
                    continue
                got = 0.0
                for wp in sample:
                    for i in sorted(set([0, nb - 1])):
                        acc = []
                        for q in (0, r - 1):
                            addr = []
                            for lane in range(32):
                                w, t = self.lane(wp * 32 + lane, cmap)
                                j = t + i * self.tpl
                                if w >= self.w or t >= self.tpl or j >= nr:
                                    addr.append(None)
                                    continue
                                k = (j - j % ns) * r + j % ns + q * ns if store else j + q * nr
                                addr.append(self.at(w, k))
                            acc.append(conflicts(addr, per))
                        got += sum(acc) / len(acc) * (nb / (1 if nb == 1 else 2))
                total += got / len(sample) * warps * r
            out.append(total)
            ns *= r
        return out

    def issue(self):
        """Warp instructions per tile of each stage, double-precision ones counted twice."""
        out, ns = [], 1
        fp = 2 if self.dbl else 1
        for s, r in enumerate(self.rs):
            first, last = s == 0, s == len(self.rs) - 1
            nr = self.n // r
            ops = FP[r] * fp + 4 * r + 10
            if not first:
                ops += fp * 4 * (2 * (r - 1) - TW_LOADS[r]) + 3 * TW_LOADS[r]
            lin = self.pads == 0 or nr % (1 << self.pads) == 0
            ops += 0 if lin or first else 2 * r
            lin = self.pads == 0 or ns % (1 << self.pads) == 0 or (1 << self.pads) % (ns * r) == 0
            ops += 0 if lin or last else 2 * r
            total = 0
            for i in range(-(-nr // self.tpl)):
                lanes = min(self.tpl, nr - i * self.tpl)
                total += ops * -(-self.w * lanes // 32)
            out.append(total)
            ns *= r
        return out

    def values(self):
        return max(-(-(self.n // r) // self.tpl) * r for r in self.rs)

    def minb(self):
        b = min(65536 // (self.threads * regs(self.values(), self.dbl)), 2048 // self.threads, 24)
        return max(1, b)

    def cost(self):
        waves = self.waves() if len(self.rs) > 1 else [0]
        size = 16 if self.dbl else 8
        blocks = min(self.minb(), SMEM // (self.w * self.pitch * size + 1024))
        if blocks < 1:
            return 1e30
        cycles = 0.0
        for s, (i, v) in enumerate(zip(self.issue(), waves)):
            r = self.rs[s]
            nb = -(-(self.n // r) // self.tpl)
            lanes = min(self.tpl, self.n // r)
            # bytes in flight of the resident blocks, of 128 KB: what hides the latencies
            held = min(1.0, blocks * self.w * lanes * nb * r * size / (1 << 17))
            cycles += (i / 4 + 0.7 * v) / held ** 0.35 + 60.0 / blocks
        return cycles / self.w * (1.06 if blocks == 1 else 1.0)


def lines(kind, dbl, n, tpl):
    """Lines per CTA to try."""
    size = 16 if dbl else 8
    if kind == KK:
        out = [w for w in (1, 2, 3, 4, 5, 6, 8, 10, 12, 16, 20, 24, 32, 48, 64) if w == 1 or w * tpl <= 288]
        if tpl >= 96:
            return out
        best = [w for w in out if w * tpl >= 96] or out[-1:]
        return best
    # segments of 64 to 128 bytes, 32 where the line does not fit otherwise
    w = 128 // size
    out = []
    while w * size >= 32:
        out.append(w)
        w //= 2
    ok = [w for w in out if w * tpl <= (512 if dbl else 1024) and w * n * size <= SMEM - 8192]
    wide = [w for w in ok if w * size >= 64 and w * tpl <= 512]
    return wide or ok[:2]


def best(dbl, kind, n, keep=KEEP):
    """The cheapest layouts under the model, best first, one per radix set, threads and lines."""
    top = max_values(dbl, kind, n)
    found = []
    least = next((s for s in range(1, 7) if multisets(n, s)), None)
    if least is None:
        return []
    least = max(least, 2)
    for stages in (least, least + 1):
        for ms in multisets(n, stages):
            lo = max(max(-(-n // top), 1), 1)
            tpls = set()
            for v in range(max(ms), top + 1):
                t = max(1, -(-n // v))
                while any(-(-(n // r) // t) * r > v for r in ms):
                    t += 1
                tpls.add(t)
            for t in tpls:
                if t < lo or t > 1024:
                    continue
                lay = Layout(dbl, kind, n, ms, t, 1, 0, n)
                found.append((sum(lay.issue()) / min(1.0, 32.0 * -(-t // 32) / t), ms, t))
    found.sort()
    result = {}
    tried = 0
    for _, ms, t in found:
        if tried >= keep + 5:
            break
        values = Layout(dbl, kind, n, ms, t, 1, 0, n).values()
        ws = [w for w in lines(kind, dbl, n, t)
              if (w * t + 31) // 32 * 32 <= min(1024, 65536 // regs(values, dbl))]
        if not ws:
            continue
        tried += 1
        orders = sorted(set(itertools.permutations(ms)))
        # an odd first radix spreads the first exchange over the banks; else the padding does
        orders.sort(key=lambda o: (o[0] % 2 == 0, -o[0]))
        for w in ws[:4]:
            for o in orders[:12]:
                for pads in (0, 3 if dbl else 4):
                    flat = n + (n >> pads) if pads else n
                    if kind == KK:
                        pitches = [flat | 1] if w > 1 else [flat]
                    else:
                        pitches = [flat + d for d in range(0, 16 if not dbl else 8)]
                        pitches = [p for p in pitches if p % (8 if dbl else 16) in ((1, 2, 4) if dbl else (1, 2, 4))]
                    for pitch in pitches:
                        lay = Layout(dbl, kind, n, o, t, w, pads, pitch)
                        if w * pitch * (16 if dbl else 8) > SMEM:
                            continue
                        c = lay.cost()
                        key = (ms, t, w)
                        if c < 1e29 and (key not in result or c < result[key][0] * (1 - 1e-9)):
                            result[key] = (c, lay)
    return [lay for _, lay in sorted(result.values(), key=lambda v: v[0])[:keep]]


# (mapping, feature, longest float line, longest double line); the real transforms of feature 2 and 4 take
# the layout chosen for the complex lines of half their length
FAMILIES = (
    (KK, 0, 16384, 8192),
    (CC, 0, 2048, 2048),
    (CC, 1, 1280, 1280),
    (CK, 0, 2048, 2048),
    (KC, 0, 2048, 2048),
)


def work(job):
    dbl, kind, n = job
    return job, best(dbl, kind, n)


def entry(l, feat):
    return "%d, %d, %d, %d, %d, %d, %d, %d, %d, %d, %s" % (
        l.dbl, l.kind, feat, l.n, l.tpl, l.w, l.pads, l.pitch, l.threads, l.minb(), ", ".join(map(str, l.rs)))


def candidates():
    """Every layout worth timing: {(dbl, kind, tw4, n): [entry text, ...]}."""
    from multiprocessing import Pool
    jobs = []
    for dbl in (0, 1):
        for kind in (KK, CC, CK, KC):
            limit = max(f[2 + dbl] for f in FAMILIES if f[0] == kind)
            jobs += [(dbl, kind, n) for n in range(16, limit + 1) if smooth(n)]
    with Pool() as pool:
        got = dict(pool.map(work, jobs, chunksize=4))
    out = {}
    for kind, tw4, fmax, dmax in FAMILIES:
        for dbl in (0, 1):
            for n in range(16, (dmax if dbl else fmax) + 1):
                if got.get((dbl, kind, n)):
                    out[(dbl, kind, tw4, n)] = [entry(l, tw4) for l in got[(dbl, kind, n)]]
    return out


HEAD = """// Written by gen_smooth_catalog.py: the size-specialised kernels of the 7-smooth lengths
// (smooth_kernel.cuh).
//
// X(ID, DOUBLE, KIND, FEAT, N, TPL, W, PADS, PITCH, MAXT, MINB, RADICES...)
//   KIND: 0 whole contiguous lines, 1 strided columns, 2 columns stored as rows, 3 rows stored as
//   columns; FEAT: 1 four-step twiddle on the store, 2 / 4 R2C / C2R of twice the length; TPL threads per line; W lines per CTA (KIND 0:
//   at most); shared-memory rows of PITCH elements, one padding element per 2^PADS (0: none);
//   RADICES the Stockham stages in order.
// SFB_SMOOTH_PART_<p> lists the entries that smooth_variants.cu compiles as part p.
#pragma once

"""


PIPED_HEAD = """// Written by gen_smooth_catalog.py --piped: the copy-engine-pipelined 7-smooth kernels (smooth_piped.cuh): even float
// lines of 4116 to 14400 points, those that timed at least 5% below the plain kernel of smooth_catalog.h (128 MB of
// lines).
//
// X(ID, DOUBLE, KIND, FEAT, N, TPL, W, PADS, PITCH, MAXT, MINB, RADICES...) as in smooth_catalog.h; KIND 0, W 1;
// FEAT 2: R2C of twice the length; MINB blocks fit an SM beside their copy buffers.
// SFB_SPIPED_PART_<p> lists the entries that smooth_piped_variants.cu compiles as part p.
#pragma once

"""


def write_parts(rows, out, macro, parts):
    """Row i goes to part i mod parts; ids number the entries in the order of the parts."""
    ident = 0
    for p in range(parts):
        out.write("#define %s_PART_%d(X) \\\n" % (macro, p))
        text = []
        for e in rows[p::parts]:
            text.append("    X(%d, %s)" % (ident, e))
            ident += 1
        out.write(" \\\n".join(text) + "\n\n")


def write_catalog(out, macro, parts):
    out.write("#define %s_CATALOG(X) %s\n" % (macro, " ".join("%s_PART_%d(X)" % (macro, p) for p in range(parts))))


def write(rows, out):
    out.write(HEAD)
    write_parts(rows, out, "SFB_SMOOTH", 24)
    out.write("#define SFB_SMOOTH_PARTS 24\n")
    write_catalog(out, "SFB_SMOOTH", 24)


def write_piped(rows, out):
    out.write(PIPED_HEAD)
    write_parts(rows, out, "SFB_SPIPED", 4)
    write_catalog(out, "SFB_SPIPED", 4)


def committed(name):
    """The rows of a committed catalog, in the order in which write_parts was given them."""
    with open(os.path.join(os.path.dirname(os.path.abspath(__file__)), name)) as f:
        parts = [re.findall(r"X\(\d+, ([-0-9, ]+)\)", part) for part in f.read().split("#define ")[1:] if "_PART_" in part.split("(")[0]]
    return [part[i] for i in range(max(map(len, parts))) for part in parts if i < len(part)]


def piped_candidates():
    """Pipelined forms of the plain float layouts, complex lines and R2C."""
    for n in range(4097, 16385):
        if n % 2 or not smooth(n):
            continue
        for feat in (0, 2):
            for l in best(0, KK, n):
                room = SMEM // ((n + l.pitch) * 8 + 16 + 1024)
                if l.w == 1 and room >= 1:
                    e = entry(l, feat).split(", ")
                    e[9] = str(min(int(e[9]), room))
                    yield ", ".join(e)


def main():
    args = sys.argv[1:]
    piped = args[:1] == ["--piped"]
    arg = args[piped] if len(args) > piped else ""
    put = write_piped if piped else write
    if arg == "--candidates":
        for rows in [piped_candidates()] if piped else candidates().values():
            print("\n".join(rows))
    elif arg:
        with open(arg) as f:
            put([line.strip() for line in f if line.strip()], sys.stdout)
    else:
        put(committed("smooth_piped_catalog.h" if piped else "smooth_catalog.h"), sys.stdout)


if __name__ == "__main__":
    main()
