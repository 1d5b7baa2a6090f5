"""The FP64 helpers of getm_common.cuh and the face function of
advection_passes.cuh, called through a small kernel: the error bounds their
comments state, the operands at which they leave the fast path, signed zeros,
subnormals, infinities and NaNs."""

import ctypes
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "advection_passes.cuh"

__global__ void unary_kernel(int n, const double* x, double* rcp, double* twice)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    rcp[q] = getm_rcp(x[q]);
    twice[q] = getm_twice(x[q]);
}

__global__ void div_kernel(int n, const double* x, const double* y, double* out)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < n) out[q] = getm_div(x[q], y[q]);
}

__global__ void face_kernel(int n, int scheme, const double* cfl, const double* QU, const double* dprev, const double* d,
                            const double* dnext, double* el, double* er)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < n) hx_face(hx_tvd(scheme, cfl[q], QU[q]), QU[q] > 0.0, true, QU[q], dprev[q], d[q], dnext[q], 0.0, false, el[q], er[q]);
}

extern "C" unsigned long long getm_launch_counter_add(void) { return 0; }

extern "C" int unary(int n, const double* x, double* rcp, double* twice)
{
    unary_kernel<<<(n + 127) / 128, 128>>>(n, x, rcp, twice);
    return cudaDeviceSynchronize();
}

extern "C" int quotient(int n, const double* x, const double* y, double* out)
{
    div_kernel<<<(n + 127) / 128, 128>>>(n, x, y, out);
    return cudaDeviceSynchronize();
}

extern "C" int face(int n, int scheme, const double* cfl, const double* QU, const double* dprev, const double* d,
                    const double* dnext, double* el, double* er)
{
    face_kernel<<<(n + 127) / 128, 128>>>(n, scheme, cfl, QU, dprev, d, dnext, el, er);
    return cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    from getm_gb300 import build

    d = tmp_path_factory.mktemp("fp64_helpers")
    src, out = d / "helpers.cu", d / "helpers.so"
    src.write_text(SOURCE)
    r = subprocess.run([build.nvcc(), *build.NVCC_FLAGS, "-shared", str(src), "-o", str(out)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(str(out))


def _call(f, n, nout, scalars, arrays):
    import torch

    torch.cuda.synchronize()
    given = [torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).cuda() for a in arrays]
    outs = [torch.full((n,), 7.0, dtype=torch.float64, device="cuda") for _ in range(nout)]
    torch.cuda.synchronize()
    assert f(n, *scalars, *[ctypes.c_void_p(t.data_ptr()) for t in given + outs]) == 0
    return [t.cpu().numpy() for t in outs]


SPECIAL = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 1e-310, 2.2250738585072014e-308,
                    -1.7976931348623157e308, 1.0, -3.5])


def _at_exponents(rng, biased, n=40):
    """Random mantissas and signs at the given biased exponents."""
    b = np.repeat(np.asarray(biased, dtype=np.uint64), n)
    m = rng.integers(0, 2**52, b.size, dtype=np.uint64)
    m[::n], m[1::n] = 0, 2**52 - 1
    s = rng.integers(0, 2, b.size, dtype=np.uint64)
    return (s << np.uint64(63) | b << np.uint64(52) | m).view(np.float64)


def _same(a, b):
    return (np.isnan(a) & np.isnan(b)) | ((a == b) & (np.signbit(a) == np.signbit(b)))


def test_reciprocal_and_twice(lib):
    rng = np.random.default_rng(1)
    x = np.concatenate([_at_exponents(rng, [0, 1, 2, 3, 2043, 2044, 2045, 2046]), _at_exponents(rng, range(4, 2043, 7)),
                        rng.uniform(0.5, 2.0, 200000), SPECIAL])
    rcp, twice = _call(lib.unary, x.size, 2, (), [x])
    with np.errstate(all="ignore"):
        want, dbl = 1.0 / x, x + x
    assert _same(twice, dbl).all()
    e = (x.view(np.uint64) >> np.uint64(52)) & np.uint64(0x7ff)
    fast = (e >= 2) & (e <= 2044)
    assert _same(rcp[~fast], want[~fast]).all()  # the division itself
    # two units in the last place, where the quotient is a normal number
    normal = fast & (np.abs(want) >= 2.2250738585072014e-308)
    assert (np.abs(rcp[normal] - want[normal]) <= 2 * np.spacing(np.abs(want[normal]))).all()
    assert normal.sum() > 0.9 * x.size


def test_division(lib):
    rng = np.random.default_rng(2)
    edges = [0, 1, 2, 63, 64, 65, 122, 123, 124, 1023, 1922, 1923, 1924, 1982, 1983, 1984, 2045, 2046]
    a = np.concatenate([_at_exponents(rng, edges, 6), SPECIAL])
    n, d = (v.ravel() for v in np.meshgrid(a, a))
    n = np.concatenate([n, rng.uniform(0.5, 2.0, 200000), _at_exponents(rng, range(100, 1900, 3), 20)])
    d = np.concatenate([d, rng.uniform(0.5, 2.0, 200000), _at_exponents(rng, range(100, 1900, 3), 20)[::-1]])
    (got,) = _call(lib.quotient, n.size, 1, (), [n, d])
    with np.errstate(all="ignore"):
        want = n / d
        wide = n.astype(np.longdouble) / d.astype(np.longdouble)
    en, ed = (((v.view(np.uint64) >> np.uint64(52)) & np.uint64(0x7ff)).astype(int) for v in (n, d))
    inside = (ed >= 64) & (ed <= 1983) & (n != 0) & (en >= 64) & (en <= 1983) & (abs(en - ed) <= 900)
    assert _same(got[~inside], want[~inside]).all()  # the division, and signed zeros
    # half a unit in the last place and less than 2^-6 of one beside it
    err = np.abs(got[inside].astype(np.longdouble) - wide[inside]) / np.spacing(np.abs(want[inside]))
    assert err.max() <= 0.5 + 2.0 ** -6
    assert inside.sum() > 200000


def _limiter(scheme, r, c):
    """limiters.h with fmin and fmax, which pass over a NaN."""
    if scheme == 1:
        k = 1.0 - c
        x = 0.25 * (k - 1.0 / 3.0 / k)
        return np.fmin(np.fmin(2.0 * r, np.fmax(0.0, (0.5 + x) + (0.5 - x) * r)), 2.0)
    if scheme == 2:
        return np.fmin(np.fmin(2.0 * r, 0.5 * (1.0 + r)), 2.0)
    if scheme == 3:
        x = (1.0 - 2.0 * c) / 6.0
        return np.fmin(np.fmin(2.0 * r / (c + 1e-10), (0.5 + x) + (0.5 - x) * r), 2.0 / (1.0 - c))
    if scheme == 4:
        return np.fmin(np.fmin(2.0 * r, np.fmax(1.0 + 2.0 * r, 2.0 + r) / 3.0), 2.0)
    if scheme == 5:
        return np.fmax(np.fmin(2.0 * r, 1.0), np.fmin(r, 2.0))
    return np.zeros_like(r)


@pytest.mark.parametrize("scheme", [1, 2, 3, 4, 5, 6])
def test_face(lib, scheme):
    """QU (face - west cell) and QU (face - east cell): random differences, and
    zeros, tiny and infinite ones and NaNs on either side.  A limited value takes
    about ten roundings, its two weights at most 2.5 with Courant numbers up to
    0.9: 40 u of QU times the larger of the difference and twice the limited one."""
    rng = np.random.default_rng(scheme)
    v = np.array([0.0, -0.0, 1.0, -0.25, 3.0, 1e-300, -1e-300, np.inf, -np.inf, np.nan])
    dprev, d, dnext = (x.ravel() for x in np.meshgrid(v, v, v))
    m = 20000
    dprev, d, dnext = (np.concatenate([x, rng.standard_normal(m)]) for x in (dprev, d, dnext))
    cfl = rng.uniform(0.05, 0.9, d.size)
    QU = rng.uniform(10.0, 1e5, d.size) * np.where(rng.random(d.size) < 0.5, 1, -1)
    el, er = _call(lib.face, d.size, 2, (scheme,), [cfl, QU, dprev, d, dnext])
    up = QU > 0
    with np.errstate(all="ignore"):
        du = np.where(up, dprev, dnext)
        on = np.sign(d) * np.sign(du) > 0  # (the product of two tiny differences is zero)
        dev = np.where(on, 0.5 * np.where(on, _limiter(scheme, du / d, cfl), 0.0) * (1.0 - cfl) * d, 0.0)
        want_l, want_r = QU * np.where(up, dev, d - dev), QU * np.where(up, dev - d, -dev)
        tol = 40 * 1.2e-16 * np.abs(QU) * np.fmax(np.fmax(np.abs(d), 2 * np.abs(dev)), 0.0) + 1e-305
    for got, want in ((el, want_l), (er, want_r)):
        fin = np.isfinite(want)
        with np.errstate(invalid="ignore"):
            bad = fin & ~(np.abs(got - want) <= tol)
        assert not bad.any(), [(x[bad][:3]) for x in (got, want, dprev, d, dnext, QU)]
        assert (np.isnan(got) == np.isnan(want))[~fin].all() and _same(got, want)[np.isinf(want)].all()
