"""The two forms of Distribution1D::SetFunction on the device (csrc/cdf.cuh),
one block and three launches, against the same additions on the CPU: 1024 chunks
of float64 sums, each rounding fixed by the order, so bit for bit. Sizes at both
sides of the limit between the forms (16,384), of the chunks and of the staged
tiles, several distributions, and a length that lies on the device."""
import os
import subprocess

import numpy as np
import pytest

from tensorray_b200 import build

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("cdf") / "cdf_harness")
    cmd = [build._nvcc(), "-O2", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
           "-fmad=false", os.path.join(HERE, "native", "cdf_harness.cu"), "-o", exe, "-lcudart"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        pytest.fail("nvcc failed:\n" + res.stderr[-2000:])
    return exe


def _cdf(w):
    n = len(w)
    chunk = max(1, -(-n // 1024))
    run, out = np.float64(0.0), np.empty(n, np.float64)
    part = np.float64(0.0)
    for a in range(0, n, chunk):
        x = w[a:a + chunk].astype(np.float64)
        out[a:a + chunk] = np.cumsum(np.concatenate([[part], x]))[1:]
        part = part + np.cumsum(x)[-1]
    cdf = out.astype(np.float32) * (np.float32(1.0) / np.float32(n))
    integral = cdf[-1]
    return (cdf / integral if integral > 0 else cdf), integral


@pytest.mark.parametrize("n,ndist,count", [(1, 1, -1), (7, 3, -1), (1023, 1, -1), (1025, 2, -1), (16_383, 1, -1),
                                           (16_384, 2, -1), (16_385, 2, -1), (100_003, 2, -1), (300_000, 1, -1),
                                           (20_000, 1, 16_385), (20_000, 1, 5), (300_000, 1, 299_999)])
def test_both_forms(harness, tmp_path, n, ndist, count):
    g = np.random.default_rng(n + ndist)
    w = np.where(g.random((ndist, n)) < 0.3, 0.0, g.lognormal(-3.0, 2.0, (ndist, n))).astype(np.float32)
    w[:, 0] = 1.0
    if ndist > 1:
        w[-1] = 0.0
    w.tofile(tmp_path / "w.f32")
    subprocess.run([harness, str(tmp_path / "w.f32"), str(tmp_path / "o.f32"), str(ndist), str(n), str(count)],
                   check=True, timeout=120)
    out = np.fromfile(tmp_path / "o.f32", np.float32).reshape(3, ndist * n + ndist)
    m = n if count < 0 else count
    for form in out:
        cdf, integral = form[:ndist * n].reshape(ndist, n), form[ndist * n:]
        assert (cdf[:, m:] == -1).all()
        for v in range(ndist):
            ref, total = _cdf(w[v, :m])
            assert integral[v] == total
            assert np.array_equal(cdf[v, :m], ref)
