"""The tuned mode's reciprocal and square roots (physics.cuh: rcp_f, rsqrt_f,
sqrt_f) against the exact functions over the range they are stated for, and
what they give at its ends."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest
import torch

from grace_b200 import build

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def approx(tmp_path_factory):
    if shutil.which(build.NVCC) is None:
        pytest.skip("no nvcc")
    so = str(tmp_path_factory.mktemp("approx") / "approx.so")
    subprocess.run([build.NVCC, *build.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared",
                    "-I", os.path.join(build.ROOT, "include"), "-I", os.path.join(build.HERE, "csrc"),
                    os.path.join(HERE, "approx_kernel.cu"), "-o", so], check=True)
    lib = ctypes.CDLL(so)

    def run(x):
        d = torch.from_numpy(np.ascontiguousarray(x)).to("cuda:0")
        out = [torch.empty_like(d) for _ in range(3)]
        p = [ctypes.c_void_p(t.data_ptr()) for t in (d, *out)]
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        assert lib.approx(ctypes.c_long(x.size), *p, stream) == 0
        return [t.cpu().numpy() for t in out]

    return run


def ulps(got, exact):
    """Error in units in the last place of the result; exact in 64-bit mantissas."""
    return np.abs((got.astype(np.longdouble) - exact) / np.spacing(np.abs(exact).astype(np.float64))).max()


def sample(lo, hi, n=1 << 20):
    """Mantissas at random and at both ends of the binade, every exponent from lo to hi."""
    rng = np.random.default_rng(3)
    m = np.concatenate([rng.uniform(1.0, 2.0, n), 1.0 + np.arange(512) * 2.0 ** -52, 2.0 - np.arange(1, 513) * 2.0 ** -52])
    e = np.concatenate([rng.integers(lo, hi, n, endpoint=True), rng.integers(lo, hi, 1024, endpoint=True)])
    return np.ldexp(m, e)


def test_approximations_over_the_normal_range(approx):
    """Within 1 (rcp_f) and 2 (rsqrt_f, sqrt_f) units in the last place: the
    correction's truncation is below 2^-54, its last operation rounds once, and
    the roots' residual carries the rounding of x y."""
    one = np.longdouble(1)
    x = sample(-1022, 1020)  # 1/x normal
    rcp, rsq, _ = approx(x)
    assert ulps(rcp, one / x.astype(np.longdouble)) <= 1.0
    assert ulps(rsq, one / np.sqrt(x.astype(np.longdouble))) <= 2.0
    rcp, _, _ = approx(-x)
    assert ulps(rcp, -one / x.astype(np.longdouble)) <= 1.0
    x = sample(-960, 1023)  # above 1e-290
    _, rsq, sq = approx(x)
    assert ulps(rsq, one / np.sqrt(x.astype(np.longdouble))) <= 2.0
    assert ulps(sq, np.sqrt(x.astype(np.longdouble))) <= 2.0


def test_approximations_at_the_ends(approx):
    """What the comment states: NaN at 0, infinity and NaN, for rcp_f at
    subnormals and where 1/x is subnormal no value to rely on, sqrt_f 0 at 0
    and below 1e-145 at what lies below 1e-290."""
    x = np.array([0.0, -0.0, np.inf, np.nan])
    rcp, rsq, sq = approx(x)
    assert np.all(np.isnan(rcp)) and np.all(np.isnan(rsq))
    assert sq[0] == 0.0 and sq[1] == 0.0 and np.all(np.isnan(sq[2:]))
    tiny = np.array([5e-324, 1e-310, 1e-300, 9e-291])
    _, _, sq = approx(tiny)
    assert np.all(sq >= 0.0) and np.all(sq < 1e-145)
    _, rsq, _ = approx(np.array([-1.0, -np.inf]))
    assert np.all(np.isnan(rsq))
