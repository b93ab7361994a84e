"""Loaders for the test-only host libraries in tests/native (built with its Makefile)."""
import ctypes
import json
import os
import subprocess

import numpy as np

HERE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native")
_cache = {}


def _load(name):
    if name not in _cache:
        subprocess.run(["make", "-s", "-C", HERE], check=True)
        _cache[name] = ctypes.CDLL(os.path.join(HERE, name))
    return _cache[name]


def butterfly(radix, x, double=True):
    L = _load("libbutterfly_check.so")
    dt = np.float64 if double else np.float32
    xin = np.ascontiguousarray(np.stack([x.real, x.imag], -1).reshape(-1).astype(dt))
    out = np.zeros_like(xin)
    fn = L.sfb_check_dft_f64 if double else L.sfb_check_dft_f32
    rc = fn(int(radix), ctypes.c_void_p(xin.ctypes.data), ctypes.c_void_p(out.ctypes.data))
    assert rc == 0
    return out[0::2] + 1j * out[1::2]


def twiddle_powers(mode, radix, w, x, double=True):
    """u[r] * w^r (r = 1..radix-1, u[0] unchanged) through the size-specialised kernels'
    twiddle_powers (mode 0: the balanced product tree)."""
    L = _load("libbutterfly_check.so")
    dt = np.float64 if double else np.float32
    xin = np.ascontiguousarray(np.stack([x.real, x.imag], -1).reshape(-1).astype(dt))
    out = np.zeros_like(xin)
    fn = L.sfb_check_powers_f64 if double else L.sfb_check_powers_f32
    real = ctypes.c_double if double else ctypes.c_float
    fn.argtypes = [ctypes.c_int, ctypes.c_int, real, real, ctypes.c_void_p, ctypes.c_void_p]
    rc = fn(int(mode), int(radix), w.real, w.imag, ctypes.c_void_p(xin.ctypes.data), ctypes.c_void_p(out.ctypes.data))
    assert rc == 0
    return out[0::2] + 1j * out[1::2]


def emulate(x, shape, batch, direction, norm=0, double=False, in_place=False, force_maxv=0, smem_limit=0):
    """Run a plan through the FP64 pass emulator; returns (output, plan description)."""
    L = _load("libplan_emulator.so")
    L.emu_run.argtypes = [ctypes.c_int] * 4 + [ctypes.c_uint, ctypes.c_void_p, ctypes.c_uint64, ctypes.c_int,
                                               ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_char_p,
                                               ctypes.c_size_t, ctypes.c_char_p, ctypes.c_size_t]
    sh = (ctypes.c_uint64 * 3)(*(list(shape) + [0] * (3 - len(shape))))
    xin = np.ascontiguousarray(np.asarray(x, dtype=np.complex128))
    out = np.zeros_like(xin)
    desc = ctypes.create_string_buffer(1 << 18)
    err = ctypes.create_string_buffer(1024)
    rc = L.emu_run(int(double), int(direction), int(norm), int(in_place), len(shape), sh, int(batch),
                   int(force_maxv), int(smem_limit), xin.ctypes.data, out.ctypes.data, desc, 1 << 18, err, 1024)
    if rc:
        raise RuntimeError(err.value.decode())
    return out, json.loads(desc.value.decode())


def emulate_skip(x, shape, batch, direction, skip_axes, norm=0, double=False, in_place=False):
    """emulate() with the axes in the bit mask `skip_axes` left untransformed."""
    L = _load("libplan_emulator.so")
    L.emu_run_skip.argtypes = [ctypes.c_int] * 4 + [ctypes.c_uint, ctypes.c_void_p, ctypes.c_uint64, ctypes.c_uint,
                                                    ctypes.c_void_p, ctypes.c_void_p, ctypes.c_char_p,
                                                    ctypes.c_size_t, ctypes.c_char_p, ctypes.c_size_t]
    sh = (ctypes.c_uint64 * 3)(*(list(shape) + [0] * (3 - len(shape))))
    xin = np.ascontiguousarray(np.asarray(x, dtype=np.complex128))
    out = np.zeros_like(xin)
    desc = ctypes.create_string_buffer(1 << 18)
    err = ctypes.create_string_buffer(1024)
    rc = L.emu_run_skip(int(double), int(direction), int(norm), int(in_place), len(shape), sh, int(batch),
                        int(skip_axes), xin.ctypes.data, out.ctypes.data, desc, 1 << 18, err, 1024)
    if rc:
        raise RuntimeError(err.value.decode())
    return out, json.loads(desc.value.decode())


def describe(shape, batch, direction=-1, norm=0, double=False, in_place=False, smem_limit=232448, split_bf16=False):
    """The planner's plan for a request (no execution), as the provider describes it."""
    L = _load("libplan_emulator.so")
    L.emu_describe.argtypes = [ctypes.c_int] * 4 + [ctypes.c_uint, ctypes.c_void_p, ctypes.c_uint64, ctypes.c_int,
                                                    ctypes.c_int, ctypes.c_int, ctypes.c_char_p, ctypes.c_size_t,
                                                    ctypes.c_char_p, ctypes.c_size_t]
    sh = (ctypes.c_uint64 * 3)(*(list(shape) + [0] * (3 - len(shape))))
    desc = ctypes.create_string_buffer(1 << 18)
    err = ctypes.create_string_buffer(1024)
    rc = L.emu_describe(int(double), direction, norm, int(in_place), len(shape), sh, batch, 0, smem_limit,
                        int(split_bf16), desc, len(desc), err, len(err))
    if rc != 0:
        raise ValueError(err.value.decode())
    return json.loads(desc.value.decode())


def primitive_root(p):
    """The planner's primitive root mod the prime p (the generator of its Rader tables)."""
    L = _load("libplan_emulator.so")
    L.emu_primitive_root.restype = ctypes.c_uint64
    L.emu_primitive_root.argtypes = [ctypes.c_uint64]
    return int(L.emu_primitive_root(int(p)))


def smooth_run(x, shape, batch, direction, norm=0, double=False, in_place=False, w_lines=0):
    """A contiguous plan stepped through the 7-smooth kernels' index arithmetic; None when a pass of the
    plan is not one of them."""
    L = _load("libsmooth_check.so")
    L.smooth_run.argtypes = [ctypes.c_int] * 4 + [ctypes.c_uint, ctypes.c_void_p, ctypes.c_uint64, ctypes.c_int,
                                                  ctypes.c_void_p, ctypes.c_void_p, ctypes.c_char_p, ctypes.c_size_t]
    sh = (ctypes.c_uint64 * 3)(*(list(shape) + [0] * (3 - len(shape))))
    xin = np.ascontiguousarray(np.asarray(x, dtype=np.complex128))
    out = np.zeros_like(xin)
    err = ctypes.create_string_buffer(1024)
    rc = L.smooth_run(int(double), int(direction), int(norm), int(in_place), len(shape), sh, int(batch), int(w_lines),
                      xin.ctypes.data, out.ctypes.data, err, 1024)
    if rc == 1:
        raise RuntimeError(err.value.decode())
    return None if rc == 2 else out


def smooth_run_line(x, n, batch, layout, out, direction, norm=0, double=False, in_place=False):
    """A strided one-dimensional plan (layout: (in cs, in ks, out cs, out ks)) likewise; writes into a copy
    of `out`."""
    L = _load("libsmooth_check.so")
    L.smooth_run_line.argtypes = [ctypes.c_int] * 4 + [ctypes.c_uint64, ctypes.c_uint64, ctypes.c_void_p, ctypes.c_void_p,
                                                       ctypes.c_int64, ctypes.c_void_p, ctypes.c_int64, ctypes.c_char_p,
                                                       ctypes.c_size_t]
    lay = (ctypes.c_int64 * 4)(*layout)
    xin = np.ascontiguousarray(np.asarray(x, dtype=np.complex128))
    got = np.array(out, dtype=np.complex128)
    err = ctypes.create_string_buffer(1024)
    rc = L.smooth_run_line(int(double), int(direction), int(norm), int(in_place), int(n), int(batch), lay,
                           xin.ctypes.data, xin.size, got.ctypes.data, got.size, err, 1024)
    if rc:
        raise RuntimeError(err.value.decode() or "no single-pass kernel")
    return got


def real_pair(pre, a, c, w, half=0.5):
    """The two bins of a real-transform pair through the kernels' pair functions."""
    L = _load("libbutterfly_check.so")
    L.sfb_check_real_pair.argtypes = [ctypes.c_int, ctypes.c_double, ctypes.c_void_p, ctypes.c_void_p]
    L.sfb_check_real_pair.restype = None
    xin = np.array([a.real, a.imag, c.real, c.imag, w.real, w.imag])
    out = np.zeros(4)
    L.sfb_check_real_pair(int(pre), float(half), xin.ctypes.data, out.ctypes.data)
    return out[0] + 1j * out[1], out[2] + 1j * out[3]


def narrow_lines(kind, feat, w, n_cols, n_outer):
    """(outer, column) of every line of column tiles that run on across outer indices, in tile order; None
    where the tiles end with the columns."""
    L = _load("libnarrow_check.so")
    L.narrow_lines.restype = ctypes.c_int64
    L.narrow_lines.argtypes = [ctypes.c_int] * 3 + [ctypes.c_int64] * 2 + [ctypes.c_void_p] * 2
    o, c = np.zeros(n_cols * n_outer, np.int64), np.zeros(n_cols * n_outer, np.int64)
    n = L.narrow_lines(kind, feat, w, n_cols, n_outer, o.ctypes.data, c.ctypes.data)
    return None if n < 0 else (o[:n], c[:n])


def tables_left_out(shape, batch, double=False, fused=False):
    """Tables of the plan that no kernel reads and that are therefore not made; asserts that the others are."""
    L = _load("libtables_check.so")
    L.tables_left_out.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_uint, ctypes.c_void_p, ctypes.c_uint64, ctypes.c_char_p,
                                  ctypes.c_size_t]
    sh = (ctypes.c_uint64 * 3)(*(list(shape) + [0] * (3 - len(shape))))
    why = ctypes.create_string_buffer(256)
    n = L.tables_left_out(int(double), int(fused), len(shape), sh, batch, why, 256)
    assert n >= 0, (shape, batch, double, why.value.decode())
    return n
