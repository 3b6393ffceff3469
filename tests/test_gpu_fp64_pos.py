"""The reciprocal, square root and threshold test that the diagnostics' FP64
terms use in place of CUDA's (csrc/fp64_pos.cuh), compiled into a small library
of their own and compared with numpy's correctly rounded 1/d and sqrt(d)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SRC = r"""
#include "fp64_pos.cuh"
__global__ void pos_kernel(const double *d, const double *t, double scale, double *recip, double *root, unsigned char *reaches, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    recip[i] = axs::recip_pos(d[i]);
    root[i] = axs::sqrt_pos(d[i]);
    reaches[i] = axs::root_reaches(d[i], scale, t[i]);
}
extern "C" int pos_run(const double *d, const double *t, double scale, double *recip, double *root, unsigned char *reaches, int n)
{
    pos_kernel<<<(n + 255) / 256, 256>>>(d, t, scale, recip, root, reaches, n);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def pos(axs, tmp_path_factory):
    from axion_strings_adaptive_gb300 import _build as B
    d = tmp_path_factory.mktemp("pos")
    (d / "pos.cu").write_text(SRC)
    r = subprocess.run([B.nvcc(), *B.ARCH_FLAGS, *B.NVCC_FLAGS, "-I", B.CSRC, "-shared", "-o", str(d / "pos.so"),
                        str(d / "pos.cu")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = C.CDLL(os.path.join(str(d), "pos.so"))

    def run(vals, thresholds, scale):
        dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (vals, thresholds)]
        n = vals.size
        out = [torch.empty(n, dtype=t, device="cuda") for t in (torch.float64, torch.float64, torch.uint8)]
        assert lib.pos_run(*[C.c_void_p(t.data_ptr()) for t in dev], C.c_double(scale),
                           *[C.c_void_p(t.data_ptr()) for t in out], C.c_int(n)) == 0
        return [t.cpu().numpy() for t in out]
    return run


def _values(kind):
    rng = np.random.default_rng(4)
    n = 1 << 20
    if kind == "physical":
        return rng.uniform(1e-6, 40.0, n)
    if kind == "float-sized":  # both sides of 2^-100 and 2^100, the float range's insides
        return np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(-104, 104, n))
    if kind == "next to a tie":  # roots for which sqrt_pos alone is an ulp off, times powers of 4
        v = np.array([0x4003084b12ad235a, 0x4003d979ec406ba3, 0x400a17eba09063d1, 0x4007ec27aa9b2b25, 0x400e68c121ec6afd,
                      0x3ff80d477ceed2b1, 0x400ead32db05f65e, 0x3ff4af74721e7211, 0x400184ab7785c523,
                      0x3ff0e85e336cc7a4, 0x3ff5611b8a535733, 0x3ff8f5e844b4cb04], dtype=np.int64).view(np.float64)
        return np.ldexp(v, 2 * np.arange(-4, 5)[:, None]).reshape(-1)
    v = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(-1060, 1023, n))  # subnormals among them
    v[:8] = [5e-324, 2.2250738585072014e-308, 2.0 ** -101, 2.0 ** -100, 2.0 ** 99, 2.0 ** 100, 1.7976931348623157e308, 1.0]
    return v


@pytest.mark.parametrize("kind", ["physical", "float-sized", "every"])
def test_reciprocal_and_root_are_within_an_ulp(pos, kind):
    """The last operation of either rounds a value within 2^-7 ulp of the true one,
    so the result is the correctly rounded one or, next to a tie, its neighbour: an
    ulp off at most, and that for less than 2^-6 of the values."""
    d = _values(kind)
    recip, root, _ = pos(d, np.ones_like(d), 1.0)
    with np.errstate(over="ignore"):
        for got, want in ((recip, 1.0 / d), (root, np.sqrt(d))):
            steps = np.abs(got.view(np.int64) - want.view(np.int64))  # positive doubles: ulps apart
            assert steps.max() <= 1 and (steps > 0).mean() < 2.0 ** -6


@pytest.mark.parametrize("scale", [1.0, 0.7])
@pytest.mark.parametrize("kind", ["physical", "float-sized", "every", "next to a tie"])
def test_threshold_decides_as_the_rounded_root(pos, kind, scale):
    d = _values(kind)
    at = np.sqrt(d) * scale
    for t in (at, np.nextafter(at, np.inf), np.nextafter(at, 0.0), at * (1 + 1e-6), at * (1 - 1e-6), -at, np.zeros_like(at)):
        assert np.array_equal(pos(d, t, scale)[2].astype(bool), at >= t)
