"""GPU parity of the size-specialised kernels of the 7-smooth lengths (smooth_kernel.cuh): the shortest and
longest lines of each thread mapping and lines per block cut off by the batch, against FP64 FFTs at the
complex tolerance of the length (rel-L2 <= 1e-5 * log2 N float, 1e-12 * log2 N double)."""
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
