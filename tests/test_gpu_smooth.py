"""GPU parity of the size-specialised kernels of the 7-smooth lengths (smooth_kernel.cuh): the shortest and
longest lines of each thread mapping, lines per block cut off by the batch, and strided layouts, against
FP64 FFTs at the complex tolerance of the length (rel-L2 <= 1e-5 * log2 N float, 1e-12 * log2 N double)."""
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


def tol(n, dbl):
    return (1e-12 if dbl else 1e-5) * max(1.0, np.log2(n))


@pytest.mark.parametrize("dbl", [False, True], ids=["float", "double"])
@pytest.mark.parametrize("shape,batch", [
    ([18], 1), ([18], 1000), ([45], 63), ([105], 25), ([343], 1), ([1000], 7), ([2187], 3), ([3000], 149), ([6125], 2),
    ([7500], 5), ([8000], 3), ([9000], 2), ([10206], 3), ([12000], 2), ([15625], 2), ([16200], 1), ([16807], 3),
    ([30000], 2), ([117649], 2), ([680400], 1), ([48, 343], 3), ([36, 2025], 1), ([35, 84, 98], 2), ([24, 2000], 2),
], ids=str)
def test_contiguous(sf, torch, shape, batch, dbl):
    n = int(np.prod(shape))
    x = uniform_complex(n * batch, n + batch, np.complex128 if dbl else np.complex64)
    for d, norm, in_place in ((-1, 0, False), (1, 3, True)):
        opts = sf.plan_options(placement=sf.placement.in_place if in_place else sf.placement.out_of_place,
                               normalization=sf.normalization(norm))
        p = sf.plan_many_dft("double" if dbl else "float", shape, batch, sf.direction(d), opts)
        a = torch.from_numpy(x).cuda()
        o = a if in_place else torch.full_like(a, 9.0)
        (p.execute(a) if in_place else p.execute(a, o)).synchronize()
        assert rel_l2(o.cpu().numpy(), fp64_fft(x, shape, batch, d, norm_scale(norm, d, n))) <= tol(n, dbl)


@pytest.mark.parametrize("shape,batch", [
    ([324], 1), ([324], 700), ([500], 301), ([1024], 13), ([945], 7), ([2401], 5), ([6000], 3), ([12288], 2), ([291600], 2),
    ([810, 24], 2), ([1024, 20], 3),
], ids=str)
def test_wide_radices(sf, torch, shape, batch):
    """Radices above 16: two and three stages of a line, columns, both passes of a four-step."""
    n = int(np.prod(shape))
    x = uniform_complex(n * batch, n + batch, np.complex64)
    for d, norm in ((-1, 0), (1, 3)):
        p = sf.plan_many_dft("float", shape, batch, sf.direction(d), sf.plan_options(normalization=sf.normalization(norm)))
        a = torch.from_numpy(x).cuda()
        o = torch.full_like(a, 9.0)
        p.execute(a, o).synchronize()
        assert rel_l2(o.cpu().numpy(), fp64_fft(x, shape, batch, d, norm_scale(norm, d, n))) <= tol(n, False)


@pytest.mark.parametrize("dbl", [False, True], ids=["float", "double"])
@pytest.mark.parametrize("n,b,src,dst", [
    (64, 24, (1, 24), (64, 1)), (64, 1, (1, 5), (64, 1)), (60, 7, (1, 9), (1, 11)), (100, 5, (107, 1), (103, 1)),
    (2048, 3, (1, 3), (2050, 1)), (1000, 17, (1001, 1), (1, 17)), (24, 33, (1, 2), (24, 1)), (1500, 9, (1, 9), (1500, 1)),
    (1920, 130, (1, 131), (1, 130)),
], ids=str)
def test_strided_lines(sf, torch, n, b, src, dst, dbl):
    """One launch for lines whose sides are contiguous (of any pitch) or adjacent columns; partial batches;
    nothing outside the output layout is written."""
    import ctypes
    from syclfft_b200 import _provider
    at_in = np.arange(b)[:, None] * src[0] + np.arange(n)[None, :] * src[1]
    at_out = np.arange(b)[:, None] * dst[0] + np.arange(n)[None, :] * dst[1]
    x = uniform_complex(int(at_in.max()) + 1, n + b, np.complex128 if dbl else np.complex64)
    lay = sf.data_layout((src[1],), src[0], (dst[1],), dst[0])
    p = sf.plan_many_dft("double" if dbl else "float", [n], b, sf.direction.forward, layout=lay)
    assert p.launches() == 1 and p.describe()["layout"]["direct"] == 1
    a = torch.from_numpy(x).cuda()
    ref = np.fft.fft(x[at_in].astype(np.complex128))
    for part in (b, max(1, b - 2)):
        o = torch.full((int(at_out.max()) + 1,), 3 - 5j, dtype=a.dtype, device="cuda")
        err = ctypes.create_string_buffer(_provider.ERR_CAP)
        rc = p._lib.syclfft_b200_execute_batch(p._handle, a.data_ptr(), o.data_ptr(), part,
                                               torch.cuda.current_stream().cuda_stream, err, _provider.ERR_CAP)
        assert rc == 0, err.value
        got = o.cpu().numpy()
        assert rel_l2(got[at_out[:part]], ref[:part]) <= tol(n, dbl)
        rest = np.ones(got.size, bool)
        rest[at_out[:part].reshape(-1)] = False
        assert np.all(got[rest] == np.complex64(3 - 5j))


@pytest.mark.parametrize("dbl", [False, True], ids=["float", "double"])
@pytest.mark.parametrize("h,batch", [(16, 5), (45, 97), (64, 3), (105, 26), (1000, 3), (2187, 2), (4096, 2), (6125, 2), (8000, 2),
                                     (13440, 2), (15625, 1)], ids=str)
def test_real_one_pass(sf, torch, h, batch, dbl):
    """Real transforms of length 2h in one launch, odd and even half lengths, against FP64 rfft / irfft; the
    imaginary parts of bins 0 and h do not matter."""
    n = 2 * h
    rt, ct = (np.float64, np.complex128) if dbl else (np.float32, np.complex64)
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, (batch, n)).astype(rt)
    fits = not dbl or h <= 8192
    opts = sf.plan_options(normalization=sf.normalization.orthogonal)
    f = sf.plan_dft_r2c_1d("double" if dbl else "float", n, batch, opts)
    b = sf.plan_dft_c2r_1d("double" if dbl else "float", n, batch, opts)
    if fits:
        assert f.launches() == 1 and b.launches() == 1
    spec = torch.full((batch * (h + 1),), 9.0, dtype=f.dtype, device="cuda")
    f.execute(torch.from_numpy(x).cuda(), spec).synchronize()
    ref = np.fft.rfft(x.astype(np.float64), axis=1, norm="ortho")
    assert rel_l2(spec.cpu().numpy(), ref.reshape(-1)) <= tol(n, dbl)
    s = ref.astype(ct)
    s[:, 0] += 3j
    s[:, h] -= 2j
    back = torch.full((batch * n,), 9.0, dtype=b.real_dtype, device="cuda")
    b.execute(torch.from_numpy(s).cuda(), back).synchronize()
    assert rel_l2(back.cpu().numpy(), x.reshape(-1).astype(np.float64)) <= 2 * tol(n, dbl)


# just above one line per SM, several lines per block with a remainder; the shortest and longest entries
@pytest.mark.parametrize("n,batch", [(4116, 301), (5488, 149), (9000, 1000), (12544, 297), (14400, 150)])
def test_pipelined_lines(sf, torch, n, batch):
    """More lines than SMs on the pipelined kernels, out of place, in place and in the other direction; buffers
    off a 16-byte boundary and a few lines of the same plan on the plain ones."""
    x = uniform_complex(n * batch, n, np.complex64)
    for d, norm, in_place in ((-1, 0, False), (1, 3, True)):
        opts = sf.plan_options(placement=sf.placement.in_place if in_place else sf.placement.out_of_place,
                               normalization=sf.normalization(norm))
        p = sf.plan_many_dft("float", [n], batch, sf.direction(d), opts)
        assert p.describe()["passes"][0]["spiped_id"] >= 0
        ref = fp64_fft(x, [n], batch, d, norm_scale(norm, d, n))
        for off in (0, 1):
            a = torch.zeros(n * batch + 1, dtype=torch.complex64, device="cuda")[off:off + n * batch]
            a.copy_(torch.from_numpy(x))
            o = a if in_place else torch.zeros(n * batch + 1, dtype=torch.complex64, device="cuda")[off:off + n * batch]
            (p.execute(a) if in_place else p.execute(a, o)).synchronize()
            assert rel_l2(o.cpu().numpy(), ref) <= tol(n, False)


@pytest.mark.parametrize("h,batch", [(4116, 149), (12544, 301), (13440, 150)])
def test_pipelined_real(sf, torch, h, batch):
    x = np.random.default_rng(h).uniform(-1, 1, (batch, 2 * h)).astype(np.float32)
    p = sf.plan_dft_r2c_1d("float", 2 * h, batch, sf.plan_options(normalization=sf.normalization(0)))
    o = torch.full((batch, h + 1), 9.0, dtype=torch.complex64, device="cuda")
    p.execute(torch.from_numpy(x).cuda(), o).synchronize()
    assert rel_l2(o.cpu().numpy(), np.fft.rfft(x.astype(np.float64), axis=-1)) <= tol(2 * h, False)


@pytest.mark.parametrize("dbl", [False, True], ids=["float", "double"])
@pytest.mark.parametrize("shape,batch", [
    ([18, 2], 1), ([18, 2], 9), ([64, 3], 5), ([375, 2], 3), ([448, 2], 4), ([500, 3], 7), ([810, 7], 3), ([1024, 2], 2),
    ([1029, 3], 3), ([100, 15], 4), ([2048, 2], 5), ([2048, 1], 3), ([20, 30, 2], 3), ([7, 25, 5], 2), ([175, 2], 301),
], ids=str)
def test_narrow_arrays(sf, torch, shape, batch, dbl):
    """Column passes over arrays narrower than a tile, whose tiles run on across outer indices: partial last
    tiles, in place and out of place, nothing outside the array written, and a smaller batch of the plan."""
    n = int(np.prod(shape))
    x = uniform_complex(n * batch, n + batch, np.complex128 if dbl else np.complex64)
    for d, norm, in_place in ((-1, 0, False), (1, 3, True)):
        opts = sf.plan_options(placement=sf.placement.in_place if in_place else sf.placement.out_of_place,
                               normalization=sf.normalization(norm))
        p = sf.plan_many_dft("double" if dbl else "float", shape, batch, sf.direction(d), opts)
        a = torch.from_numpy(x).cuda()
        big = torch.full((n * (batch + 2),), 9.0, dtype=a.dtype, device="cuda")
        o = big[n:n * (batch + 1)]
        if in_place:
            o.copy_(a)
        (p.execute(o) if in_place else p.execute(a, o)).synchronize()
        ref = fp64_fft(x, shape, batch, d, norm_scale(norm, d, n))
        assert rel_l2(o.cpu().numpy(), ref) <= tol(n, dbl)
        assert torch.all(big[:n] == 9.0) and torch.all(big[n * (batch + 1):] == 9.0)
        if batch > 1 and not in_place:
            big.fill_(9.0)
            import ctypes
            from syclfft_b200 import _provider
            err = ctypes.create_string_buffer(_provider.ERR_CAP)
            rc = p._lib.syclfft_b200_execute_batch(p._handle, a.data_ptr(), big.data_ptr(), batch - 1,
                                                   torch.cuda.current_stream().cuda_stream, err, _provider.ERR_CAP)
            assert rc == 0, err.value
            got = big.cpu().numpy()
            assert rel_l2(got[:n * (batch - 1)], ref[:n * (batch - 1)]) <= tol(n, dbl)
            assert np.all(got[n * (batch - 1):] == 9.0)


@pytest.mark.parametrize("n,batch,dbl,kind", [(1458, 5, False, "c2c"), (1372, 3, True, "c2c"), (9408, 150, False, "c2c"), (2861, 3, False, "c2c"),
                                              (26 * 525, 2, False, "r2c"), (9000, 2, True, "c2c")], ids=str)
def test_first_execute_under_capture(sf, torch, n, batch, dbl, kind):
    """A plan loads its kernels when it is made, so that its very first execute can be captured."""
    s = "double" if dbl else "float"
    if kind == "r2c":
        x = np.random.default_rng(n).uniform(-1, 1, (batch, n)).astype(np.float32)
        p = sf.plan_dft_r2c_1d(s, n, batch)
        ref = np.fft.rfft(x.astype(np.float64), axis=1)
    else:
        x = uniform_complex(n * batch, n, np.complex128 if dbl else np.complex64)
        p = sf.plan_many_dft(s, [n], batch, sf.direction.forward)
        ref = fp64_fft(x, [n], batch, -1)
    a = torch.from_numpy(x).cuda()
    o = torch.zeros(ref.shape, dtype=torch.complex128 if dbl else torch.complex64, device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        p.execute(a, o)
    assert torch.count_nonzero(o) == 0
    g.replay()
    torch.cuda.synchronize()
    assert rel_l2(o.cpu().numpy(), ref) <= tol(n, dbl)
    del g
