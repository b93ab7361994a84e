"""planning_mode::measure of plans that have a one-pass and a multi-pass form: strided one-dimensional layouts and
real transforms. Both forms are timed, the report names the choice, and either choice computes the transform."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import rel_l2, uniform_complex

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


def tol(n):
    return 1e-5 * np.log2(n)


def check_report(tuning):
    assert tuning["choice"] in ("one_pass", "multi_pass")
    if not tuning.get("cached"):
        ms = tuning["candidates"]
        assert set(ms) == {"one_pass", "multi_pass"} and min(ms.values()) > 0
        assert tuning["choice"] == min(ms, key=ms.get)


# columns to rows of a matrix; lines of a pitch, in place; columns of more than the tuner's 256 MB (timed on fewer)
@pytest.mark.parametrize("n,b,src,dst,in_place", [
    (360, 200, (1, 200), (360, 1), False), (256, 64, (300, 1), (300, 1), True), (1024, 40000, (1, 40000), (1024, 1), False),
], ids=str)
def test_strided_lines_are_tuned(sf, torch, n, b, src, dst, in_place):
    opts = sf.plan_options(planning=sf.planning_mode.measure,
                           placement=sf.placement.in_place if in_place else sf.placement.out_of_place)
    lay = sf.data_layout((src[1],), src[0], (dst[1],), dst[0])
    for again in (False, True):
        p = sf.plan_many_dft("float", [n], b, sf.direction.forward, opts, layout=lay)
        d = p.describe()
        if d["layout"]["direct"]:
            check_report(d["inner"]["tuning"])
            assert d["inner"]["tuning"]["choice"] == "one_pass" and bool(d["inner"]["tuning"].get("cached")) >= again
        else:
            assert d["inner"]["tuning"]["choice"]  # the inner plan's own report
    lines = min(b, 50)
    at_in = np.arange(b)[:, None] * src[0] + np.arange(n)[None, :] * src[1]
    at_out = np.arange(b)[:, None] * dst[0] + np.arange(n)[None, :] * dst[1]
    x = uniform_complex(int(at_in.max()) + 1, n + b, np.complex64)
    a = torch.from_numpy(x).cuda()
    o = a if in_place else torch.zeros(int(at_out.max()) + 1, dtype=a.dtype, device="cuda")
    (p.execute(a) if in_place else p.execute(a, o)).synchronize()
    got = o.cpu().numpy()
    for first in (0, b - lines):
        rows = slice(first, first + lines)
        assert rel_l2(got[at_out[rows]], np.fft.fft(x[at_in[rows]].astype(np.complex128))) <= tol(n)


@pytest.mark.parametrize("kind", ["r2c", "c2r"])
def test_real_lines_are_tuned(sf, torch, kind):
    n, b = 3000, 70
    opts = sf.plan_options(planning=sf.planning_mode.measure)
    p = (sf.plan_dft_r2c_1d if kind == "r2c" else sf.plan_dft_c2r_1d)("float", n, b, opts)
    d = p.describe()
    assert d["inner"]["tuning"]["choice"]
    if d["fused"]:
        check_report(d["inner"]["tuning"])
    x = np.random.default_rng(n).uniform(-1, 1, (b, n)).astype(np.float32)
    spec = np.fft.rfft(x.astype(np.float64), axis=1)
    if kind == "r2c":
        o = torch.zeros((b, n // 2 + 1), dtype=torch.complex64, device="cuda")
        p.execute(torch.from_numpy(x).cuda(), o).synchronize()
        assert rel_l2(o.cpu().numpy(), spec) <= tol(n)
    else:
        o = torch.zeros((b, n), dtype=torch.float32, device="cuda")
        p.execute(torch.from_numpy(spec.astype(np.complex64)).cuda(), o).synchronize()
        assert rel_l2(o.cpu().numpy(), n * x.astype(np.float64)) <= tol(n)


def test_kept_choice_of_the_multi_pass_form(torch, tmp_path):
    """A choice read from the tuner's file builds that form."""
    name = torch.cuda.get_device_name(0)
    kept = tmp_path / "choices"
    kept.write_text("%s|c|oop|b20|360|layout|20,1|1,360\tmulti_pass\n%s|c|r2c|b20|3000\tmulti_pass\n" % (name, name))
    code = """
import json, sys
import numpy as np, torch
import syclfft_b200 as sf
o = sf.plan_options(planning=sf.planning_mode.measure)
p = sf.plan_many_dft("float", [360], 20, sf.direction.forward, o, layout=sf.data_layout((20,), 1, (1,), 360))
x = np.random.default_rng(1).uniform(-1, 1, (360, 20)).astype(np.complex64)
y = torch.zeros((20, 360), dtype=torch.complex64, device="cuda")
p.execute(torch.from_numpy(x).cuda(), y).synchronize()
e = np.linalg.norm(y.cpu().numpy() - np.fft.fft(x.T.astype(np.complex128))) / np.linalg.norm(np.fft.fft(x.T))
q = sf.plan_dft_r2c_1d("float", 3000, 20, o)
r = np.random.default_rng(2).uniform(-1, 1, (20, 3000)).astype(np.float32)
z = torch.zeros((20, 1501), dtype=torch.complex64, device="cuda")
q.execute(torch.from_numpy(r).cuda(), z).synchronize()
f = np.linalg.norm(z.cpu().numpy() - np.fft.rfft(r.astype(np.float64))) / np.linalg.norm(np.fft.rfft(r))
print(json.dumps([p.describe()["layout"]["direct"], p.launches(), e, q.describe()["fused"], q.launches(), f]))
"""
    env = dict(os.environ, SYCLFFT_B200_TUNE_CACHE=str(kept), PYTHONPATH=os.pathsep.join(sys.path))
    run = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stderr[-2000:]
    direct, launches, e, fused, real_launches, f = json.loads(run.stdout.strip().splitlines()[-1])
    assert direct == 0 and launches >= 2 and e <= tol(360)
    assert fused == 0 and real_launches >= 2 and f <= tol(3000)
