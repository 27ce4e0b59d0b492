"""Float64 products, reciprocals and quotients in integers (swb_f64.cuh) against
the host's IEEE operations, in a kernel of their own: significands at the ends
and in the middle, ties, quotients at the bottom of a binade, the whole exponent
range, signed zeros and numbers that are not finite.  Bits are equal wherever the
integers hold the numbers, and they hold what their comments say they do."""
import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest

import swalbe_gb300  # noqa: F401  (its build module is hidden by the function of that name)

B = sys.modules["swalbe_gb300.build"]
pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "swb_f64.cuh"
using namespace swb;
// out: mul64<true>, mul64<false>, quot64; bad: a bit of each; rec: recip64(b)
__global__ void ops(const double *a, const double *b, int n, double *out, int *bad, unsigned long long *rec) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    bool p = false, q = false, d = false;
    out[i] = mul64<true>(a[i], b[i], p);
    out[n + i] = mul64<false>(a[i], b[i], q);
    rec[i] = recip64(b[i]);
    out[2 * n + i] = quot64(a[i], b[i], rec[i], d);
    bad[i] = (p ? 1 : 0) | (q ? 2 : 0) | (d ? 4 : 0);
}
// recip64 of the significands 1 + i 2^-23 (lo: the bits below those) for i below 2^23
__global__ void recips(unsigned lo, unsigned long long *rec) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 1u << 23) return;
    rec[i] = recip64(__hiloint2double((int)(0x3ff00000u | i >> 3), (int)(i << 29 | lo)));
}
extern "C" int run_ops(const double *a, const double *b, int n, double *out, int *bad, unsigned long long *rec) {
    double *d = nullptr;
    unsigned long long *r = nullptr;
    int *f = nullptr;
    cudaError_t e = cudaMalloc((void **)&d, (size_t)n * 5 * 8);
    if (!e) e = cudaMalloc((void **)&r, (size_t)n * 8);
    if (!e) e = cudaMalloc((void **)&f, (size_t)n * 4);
    if (!e) e = cudaMemcpy(d, a, (size_t)n * 8, cudaMemcpyHostToDevice);
    if (!e) e = cudaMemcpy(d + n, b, (size_t)n * 8, cudaMemcpyHostToDevice);
    if (!e) {
        ops<<<(n + 127) / 128, 128>>>(d, d + n, n, d + 2 * (size_t)n, f, r);
        e = cudaGetLastError();
    }
    if (!e) e = cudaMemcpy(out, d + 2 * (size_t)n, (size_t)n * 3 * 8, cudaMemcpyDeviceToHost);
    if (!e) e = cudaMemcpy(rec, r, (size_t)n * 8, cudaMemcpyDeviceToHost);
    if (!e) e = cudaMemcpy(bad, f, (size_t)n * 4, cudaMemcpyDeviceToHost);
    cudaFree(d);
    cudaFree(r);
    cudaFree(f);
    return (int)e;
}
extern "C" int run_recips(unsigned lo, unsigned long long *rec) {
    unsigned long long *r = nullptr;
    cudaError_t e = cudaMalloc((void **)&r, (size_t)8 << 23);
    if (!e) {
        recips<<<(1 << 23) / 256, 256>>>(lo, r);
        e = cudaGetLastError();
    }
    if (!e) e = cudaMemcpy(rec, r, (size_t)8 << 23, cudaMemcpyDeviceToHost);
    cudaFree(r);
    return (int)e;
}
"""


@pytest.fixture(scope="module")
def kernels(tmp_path_factory):
    d = tmp_path_factory.mktemp("f64")
    (d / "ops.cu").write_text(SOURCE)
    inc = os.path.join(os.path.dirname(B.PKG_DIR), "include")
    subprocess.check_call([B.nvcc(), *B.ARCH, *B.COMMON, *B.UNITS["swb_step_f64.cu"], "-I", B.CSRC, "-I", inc,
                           "-shared", "-o", str(d / "ops.so"), str(d / "ops.cu")])
    return C.CDLL(str(d / "ops.so"))


def ptr(a):
    return a.ctypes.data_as(C.c_void_p)


def run(k, a, b):
    n = a.size
    out, bad, rec = np.empty((3, n)), np.empty(n, np.int32), np.empty(n, np.uint64)
    assert k.run_ops(ptr(a), ptr(b), C.c_int(n), ptr(out), ptr(bad), ptr(rec)) == 0
    return out, bad, rec


def significands(kind, n, rng):
    """Pairs of 52 bits below the leading one."""
    full = (1 << 52) - 1
    r = lambda: rng.integers(0, full + 1, n, dtype=np.uint64)
    if kind == "any":
        return r(), r()
    edge = np.array([0, 1, 2, 3, full, full - 1, full - 2, 1 << 51, (1 << 51) - 1, (1 << 51) + 1, 1 << 29,
                     (1 << 29) - 1, full ^ ((1 << 29) - 1), 0x6a09e667f3bcc, 0x6a09e667f3bcd], np.uint64)
    if kind == "edges":  # all pairs, over and over
        i = np.arange(n) % edge.size ** 2
        return edge[i // edge.size], edge[i % edge.size]
    if kind == "one edge":
        return edge[rng.integers(0, edge.size, n)], r()
    if kind == "ties":  # products with few bits below the rounding position
        s = rng.integers(20, 33, n)
        x = (rng.integers(0, 1 << 33, n, dtype=np.uint64) << np.uint64(19)) & np.uint64(full)
        return x, (np.uint64(1) << s.astype(np.uint64)) * rng.integers(1, 1 << 19, n, dtype=np.uint64) & np.uint64(full)
    if kind == "near":  # quotients next to 1, at either side of a binade's end
        x = r()
        return x, np.clip(x.astype(np.int64) + rng.integers(-4, 5, n), 0, full).astype(np.uint64)
    raise ValueError(kind)


def assemble(m, e, s):
    return (m | e.astype(np.uint64) << np.uint64(52) | s.astype(np.uint64) << np.uint64(63)).view(np.float64)


def bits_equal(x, y):
    return (x.view(np.uint64) == y.view(np.uint64)) | (np.isnan(x) & np.isnan(y))


def normal(x):
    return np.isfinite(x) & (np.abs(x) >= 2.0 ** -1022)


@pytest.mark.parametrize("exponents", [(1, 2047), (900, 1150), (0, 2048), (0, 60), (1990, 2048), (1022, 1025)], ids=str)
@pytest.mark.parametrize("kind", ["any", "edges", "one edge", "ties", "near"])
def test_products_and_quotients(kernels, kind, exponents):
    rng = np.random.default_rng(11)
    n = 400_000
    ma, mb = significands(kind, n, rng)
    a, b = (assemble(m, rng.integers(*exponents, n), rng.integers(0, 2, n)) for m in (ma, mb))
    with np.errstate(all="ignore"):
        p, q = a * b, a / b
    out, bad, _ = run(kernels, a, b)
    ok = normal(a) & normal(b)
    zeros = np.isfinite(a) & np.isfinite(b) & ((a == 0) | (b == 0)) & (normal(a) | (a == 0)) & (normal(b) | (b == 0))
    for i, want in enumerate((p, p, q)):
        held = (bad >> i & 1) == 0
        assert bits_equal(out[i], want)[held].all(), i
    # what they hold: products of normal numbers that are normal and not next to either end
    inside = ok & (np.abs(p) >= 2.0 ** -1021) & (np.abs(p) < 2.0 ** 1023)
    assert not (bad[inside] & 3).any()
    assert not (bad[zeros] & 1).any()
    # and quotients that are, but for some next to a power of two
    frac = np.abs(np.frexp(q)[0])
    inside = ok & (np.abs(q) >= 2.0 ** -1021) & (np.abs(q) < 2.0 ** 1023) & (frac > 0.5 + 2.0 ** -50) & (frac < 1 - 2.0 ** -50)
    assert not (bad[inside] & 4).any()
    # anything that is not normal or zero is left to the caller
    odd = ~(normal(a) | (a == 0)) | ~(normal(b) | (b == 0))
    assert (bad[odd] & 2 != 0).all() and (bad[odd & (a != 0) & (b != 0)] & 1 != 0).all()
    assert (bad[~normal(b)] & 4 != 0).all() and (bad[~(normal(a) | (a == 0))] & 4 != 0).all()


def test_signed_zeros(kernels):
    a = np.array([0.0, -0.0, 0.0, -0.0, 1.5, -1.5, 1.5, -1.5])
    b = np.array([3.0, 3.0, -3.0, -3.0, 0.0, 0.0, -0.0, -0.0])
    out, bad, _ = run(kernels, a, b)
    assert not (bad & 1).any() and (bad & 2 != 0).all()
    assert bits_equal(out[0], a * b).all()
    assert not (bad[:4] & 4).any() and bits_equal(out[2][:4], a[:4] / b[:4]).all()
    assert (bad[4:] & 4 != 0).all()


@pytest.mark.parametrize("low", [0, 1, (1 << 28), (1 << 29) - 1])
def test_every_first_estimate(kernels, low):
    """The reciprocal's FP32 estimate sees the upper 23 bits of a significand:
    all of them, the operands next to 1 and 2 among them."""
    rec = np.empty(1 << 23, np.uint64)
    assert kernels.run_recips(C.c_uint(low), ptr(rec)) == 0
    b = (1 << 52) + (np.arange(1 << 23, dtype=np.int64) << 29) + low
    u = b.astype(np.uint64)
    # rec times the significand b is 2^115 - left, in two words of 64 bits
    lo32, w = np.uint64(0xffffffff), np.uint64(32)
    rh, rl, bh, bl = rec >> w, rec & lo32, u >> w, u & lo32
    mid = (rl * bl >> w) + (rh * bl & lo32) + (rl * bh & lo32)
    upper = rh * bh + (rh * bl >> w) + (rl * bh >> w) + (mid >> w)
    left = (np.uint64(0) - rec * u).astype(np.int64)
    assert np.array_equal(upper, np.where(left > 0, (1 << 51) - 1, 1 << 51).astype(np.uint64))
    assert (np.abs(left) <= 6 * b).all()
