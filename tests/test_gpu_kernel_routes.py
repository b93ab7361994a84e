"""Kernels that other lengths or batches than the everyday ones reach: the runtime-length kernel of contiguous lines.
FP64 references at the complex tolerance of the length."""
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
