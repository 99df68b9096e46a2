"""GPU: the reciprocals, quotients and roots of f3d_f64.cuh over the whole range of binary64 (zeros,
subnormal numbers, infinities and NaN among them) against IEEE arithmetic."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from flame3d_mhd_gb300 import build as b

pytestmark = pytest.mark.gpu

SOURCE = """
#include "f3d_f64.cuh"
using namespace f3d;
__global__ void k(const double* a, const double* b, double* out, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = recip(f64(b[i])).v;
    out[n + i] = recip_ieee(f64(b[i])).v;
    out[2 * n + i] = (f64(a[i]) / f64(b[i])).v;
    out[3 * n + i] = root(f64(a[i])).v;
    out[4 * n + i] = (f64(a[i]) + f64(b[i])).v;
    out[5 * n + i] = F64(f64(a[i]) * f64(b[i])).v;
}
extern "C" int run(const double* a, const double* b, double* out, int n) {
    k<<<(n + 255) / 256, 256>>>(a, b, out, n);
    return cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def run(gpu_lib, tmp_path_factory):
    import torch
    d = tmp_path_factory.mktemp("f64")
    (d / "f64.cu").write_text(SOURCE)
    subprocess.run([b.nvcc(), *b.ARCH, "-O3", "-std=c++17", "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-shared",
                    f"-I{b.CSRC}", "-o", str(d / "f64.so"), str(d / "f64.cu")], check=True)
    lib = C.CDLL(str(d / "f64.so"))

    def call(x, y):
        t = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (x, y)]
        out = torch.empty(6 * x.size, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        assert lib.run(*[C.c_void_p(v.data_ptr()) for v in (*t, out)], C.c_int(x.size)) == 0
        return out.cpu().numpy().reshape(6, -1)
    return call


def _numbers(r, n):
    """n patterns: all exponents and both signs, mantissas random, all zeros, all ones and nearly so"""
    m = r.integers(0, 1 << 52, n, dtype=np.int64)
    edge = r.integers(0, 8, n)
    m = np.where(edge == 0, 0, np.where(edge == 1, (1 << 52) - 1, np.where(edge == 2, m & 0xff, np.where(edge == 3, m | ~np.int64(0xff) & ((1 << 52) - 1), m))))
    e = r.integers(0, 2048, n, dtype=np.int64)
    s = r.integers(0, 2, n, dtype=np.int64)
    return ((s << 63) | (e << 52) | m).view(np.float64)


def _same(a, b):
    """equal bits, any NaN like any other"""
    return (a.view(np.int64) == b.view(np.int64)) | (np.isnan(a) & np.isnan(b))


@pytest.mark.parametrize("seed", range(4))
def test_against_ieee(run, seed):
    r = np.random.default_rng(seed)
    n = 1 << 19
    x, y = _numbers(r, n), _numbers(r, n)
    if seed >= 2:  # neighbouring exponents: quotients of order one
        ex, ey = ((v.view(np.int64) >> 52) & 2047 for v in (x, y))
        k = np.clip(ex + r.integers(-3, 4, n), 0, 2047)
        y = ((y.view(np.int64) & ~(np.int64(2047) << 52)) | (k << 52)).view(np.float64)
    rc, ri, q, rt, add, mul = run(x, y)
    with np.errstate(all="ignore"):
        one, quo, sq = 1.0 / y, x / y, np.sqrt(x)
        assert _same(add, x + y).all() and _same(mul, x * y).all()
    # corrected by one residual: within 2^-105 of the exact value before the last rounding, so that of
    # 2^21 numbers none is expected to fall on the wrong side of a rounding boundary (2^-53 of them do)
    assert _same(ri, one).all()
    assert _same(q, quo).all()
    # one reciprocal step leaves 2^-63 before the last rounding: within one unit in the last place
    near = _same(rc, one) | (np.abs(rc.view(np.int64) - one.view(np.int64)) <= 1)
    assert near.all()
    # the root's residual correction leaves 2^-85: of 2^21 roots at most one or two fall on the wrong side
    off = ~_same(rt, sq)
    assert off.sum() <= 2 and (np.abs(rt[off].view(np.int64) - sq[off].view(np.int64)) <= 1).all()
