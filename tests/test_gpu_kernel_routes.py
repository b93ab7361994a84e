"""Kernels that other lengths or batches than the everyday ones reach: the runtime-length kernel of contiguous lines,
the pipelined 7-smooth lines (their plain form for a few lines, and the copy wait that gives up), and the one-pass
real kernels of SYCLFFT_B200_REAL_FUSED=fixed. FP64 references at the complex tolerance of the length."""
import ctypes

import numpy as np
import pytest

from conftest import fp64_fft, norm_scale, rel_l2, uniform_complex

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch as t
    if not t.cuda.is_available():
        pytest.skip("no CUDA device")
    return t


@pytest.fixture(scope="module")
def sf():
    import syclfft_b200
    return syclfft_b200


def tol(n, dbl=False):
    return (1e-12 if dbl else 1e-5) * max(1.0, np.log2(n))


# lines below 16 points (a batch below a tile that is no power of two goes to the general kernel), a line no size-specialised kernel has, four-steps with a factor above 1280 (columns) or 2048
# (rows); radix-15 stages and both passes
@pytest.mark.parametrize("n,batch,dbl,kernels", [
    (6, 301, False, ["lean"]), (15, 100, False, ["general"]), (15, 128, False, ["lean"]), (14, 33, True, ["general"]), (14, 64, True, ["lean"]), (6804, 3, True, ["lean"]),
    (823543, 2, False, ["smooth", "lean"]), (1822500, 1, False, ["lean", "smooth"]), (2160900, 1, False, ["lean", "smooth"]),
    (3781575, 1, True, ["lean", "lean"]), (1 << 24, 1, False, ["lean", "lean"]),
], ids=str)
def test_runtime_length_kernel(sf, torch, n, batch, dbl, kernels):
    x = uniform_complex(n * batch, n, np.complex128 if dbl else np.complex64)
    for d, norm in ((-1, 0), (1, 3)):
        p = sf.plan_many_dft("double" if dbl else "float", [n], batch, sf.direction(d),
                             sf.plan_options(normalization=sf.normalization(norm)))
        assert [q["kernel"] for q in p.describe()["passes"]] == kernels
        a = torch.from_numpy(x).cuda()
        o = torch.full_like(a, 9.0)
        p.execute(a, o).synchronize()
        assert rel_l2(o.cpu().numpy(), fp64_fft(x, [n], batch, d, norm_scale(norm, d, n))) <= tol(n, dbl)


@pytest.mark.parametrize("few", [1, 100, 148])
def test_pipelined_plan_runs_a_few_lines(sf, torch, few):
    n, batch = 12544, 297
    p = sf.plan_many_dft("float", [n], batch, sf.direction.forward)
    assert p.describe()["passes"][0]["spiped_id"] >= 0
    x = uniform_complex(n * few, few, np.complex64)
    a = torch.from_numpy(x).cuda()
    o = torch.full((n * batch,), 9.0, dtype=a.dtype, device="cuda")
    err = ctypes.create_string_buffer(1024)
    rc = p._lib.syclfft_b200_execute_batch(p._handle, a.data_ptr(), o.data_ptr(), few,
                                           torch.cuda.current_stream().cuda_stream, err, 1024)
    assert rc == 0, err.value
    got = o.cpu().numpy()
    assert rel_l2(got[:n * few], fp64_fft(x, [n], few, -1)) <= tol(n) and np.all(got[n * few:] == 9.0)


@pytest.mark.parametrize("kind", ["c2c", "r2c"])
def test_pipelined_line_wait_that_gives_up(sf, torch, kind):
    """With a wait limit of 0 polls every block gives up its first copy wait, lets the copy land and returns: the
    event raises execution_failed once, and the default limit then computes the transform."""
    if kind == "c2c":
        n, batch = 12544, 297
        x = uniform_complex(n * batch, n, np.complex64)
        p = sf.plan_many_dft("float", [n], batch, sf.direction.forward)
        ref, out = fp64_fft(x, [n], batch, -1), (batch * n,)
    else:
        n, batch = 26880, 150
        x = np.random.default_rng(n).uniform(-1, 1, (batch, n)).astype(np.float32)
        p = sf.plan_dft_r2c_1d("float", n, batch)
        ref, out = np.fft.rfft(x.astype(np.float64), axis=1), (batch, n // 2 + 1)
    a = torch.from_numpy(x).cuda()
    o = torch.zeros(out, dtype=torch.complex64, device="cuda")
    assert p._lib.syclfft_b200_plan_set_wait_limit(p._handle, 0) == 0
    ev = p.execute(a, o)
    with pytest.raises(sf.SyclfftError) as info:
        ev.synchronize()
    assert info.value.code == sf.error_code.execution_failed
    assert p._lib.syclfft_b200_plan_status(p._handle) == 0  # reported once, then cleared
    ev.synchronize()
    assert p._lib.syclfft_b200_plan_set_wait_limit(p._handle, -1) == 0
    p.execute(a, o).synchronize()
    assert rel_l2(o.cpu().numpy(), ref) <= tol(n)


@pytest.mark.parametrize("n,dbl", [(512, False), (2048, False), (8192, False), (512, True), (4096, True)])
def test_fixed_real_kernels(sf, torch, n, dbl, monkeypatch):
    """The power-of-two one-pass real kernels that SYCLFFT_B200_REAL_FUSED=fixed asks for."""
    monkeypatch.setenv("SYCLFFT_B200_REAL_FUSED", "fixed")
    s, batch = "double" if dbl else "float", 37
    opts = sf.plan_options(normalization=sf.normalization.orthogonal)
    f, b = sf.plan_dft_r2c_1d(s, n, batch, opts), sf.plan_dft_c2r_1d(s, n, batch, opts)
    assert f.launches() == 1 and b.launches() == 1 and f.describe()["fused"] == 1
    x = np.random.default_rng(n).uniform(-1, 1, (batch, n)).astype(np.float64 if dbl else np.float32)
    spec = torch.zeros((batch, n // 2 + 1), dtype=f.dtype, device="cuda")
    back = torch.zeros((batch, n), dtype=b.real_dtype, device="cuda")
    f.execute(torch.from_numpy(x).cuda(), spec).synchronize()
    assert rel_l2(spec.cpu().numpy(), np.fft.rfft(x.astype(np.float64), axis=1, norm="ortho")) <= tol(n, dbl)
    b.execute(spec, back).synchronize()
    assert rel_l2(back.cpu().numpy(), x.astype(np.float64)) <= 2 * tol(n, dbl)
