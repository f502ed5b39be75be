"""The straight-line quotients and roots of csrc/ieee_div.cuh are IEEE 754's,
bit for bit, wherever their guard accepts the operands; numpy's are the oracle.

Operands: random ones over and beyond the guarded ranges, with random, sparse
and nearly full mantissas, and for roots every x whose root lies within 2^-45
ulp of the midpoint of two doubles (there an error below an ulp's 2^-53, which
the method allows before its last rounding, could show); for quotients, ones
whose distance from such a midpoint is a few times the least that there is; and
the approximations that both start from, at every mantissa they distinguish."""
import ctypes
import math
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "pennant-legion_b200", "csrc")

SOURCE = r"""
#include "ieee_div.cuh"
using namespace pnt;
__global__ void quots(const double* a, const double* b, long n, double* q, double* q0, double* inv, int* ok) {
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    ieee::Guard g, gz, gi;
    const double y = ieee::rcp(b[i], g);
    gz = g;
    gi = g;
    q[i] = ieee::quot(a[i], b[i], y, g);
    q0[i] = ieee::quot0(a[i], b[i], y, gz);
    inv[i] = y;
    ok[i] = (g.ok() ? 1 : 0) | (gz.ok() ? 2 : 0) | (gi.ok() ? 4 : 0);
}
__global__ void roots(const double* x, long n, double* r, int* ok) {
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    ieee::Guard g;
    r[i] = ieee::root(x[i], g);
    ok[i] = g.ok() ? 1 : 0;
}
__global__ void starts(const double* x, long n, double* y, double* z, int* ok) {
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y[i]) : "d"(x[i]));
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(z[i]) : "d"(x[i]));
    ok[i] = 1;
}
template <typename F>
static int run(int nin, const double* const* in, int nout, double* const* out, int* ok, long n, F launch) {
    double* d[8] = {};
    int* dok = nullptr;
    cudaError_t e = cudaMalloc(&dok, n * sizeof(int));
    for (int i = 0; i < nin + nout && e == cudaSuccess; ++i) {
        e = cudaMalloc(&d[i], n * 8);
        if (e == cudaSuccess && i < nin) e = cudaMemcpy(d[i], in[i], n * 8, cudaMemcpyHostToDevice);
    }
    if (e == cudaSuccess) { launch(d, dok); e = cudaDeviceSynchronize(); }
    for (int i = 0; i < nout && e == cudaSuccess; ++i) e = cudaMemcpy(out[i], d[nin + i], n * 8, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(ok, dok, n * sizeof(int), cudaMemcpyDeviceToHost);
    for (double* p : d) cudaFree(p);
    cudaFree(dok);
    return (int)e;
}
extern "C" int run_quots(const double* a, const double* b, long n, double* q, double* q0, double* inv, int* ok) {
    const double* in[2] = {a, b};
    double* out[3] = {q, q0, inv};
    return run(2, in, 3, out, ok, n, [&](double** d, int* o) { quots<<<(n + 255) / 256, 256>>>(d[0], d[1], n, d[2], d[3], d[4], o); });
}
extern "C" int run_starts(const double* x, long n, double* y, double* z, int* ok) {
    const double* in[1] = {x};
    double* out[2] = {y, z};
    return run(1, in, 2, out, ok, n, [&](double** d, int* o) { starts<<<(n + 255) / 256, 256>>>(d[0], n, d[1], d[2], o); });
}
extern "C" int run_roots(const double* x, long n, double* r, int* ok) {
    const double* in[1] = {x};
    double* out[1] = {r};
    return run(1, in, 1, out, ok, n, [&](double** d, int* o) { roots<<<(n + 255) / 256, 256>>>(d[0], n, d[1], o); });
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    d = tmp_path_factory.mktemp("ieee_div")
    (d / "t.cu").write_text(SOURCE)
    so = d / "t.so"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-fmad=false", "-std=c++17", "-shared",
                    "-Xcompiler", "-fPIC", "-I", CSRC, "-o", str(so), str(d / "t.cu")], check=True)
    return ctypes.CDLL(str(so))


def _mantissas(rng, n):
    full = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    ones = ~(rng.integers(0, 1 << 52, n, dtype=np.uint64) >> rng.integers(0, 52, n, dtype=np.uint64)) & np.uint64((1 << 52) - 1)
    sparse = (np.uint64(1) << rng.integers(0, 52, n, dtype=np.uint64)) | (np.uint64(1) << rng.integers(0, 52, n, dtype=np.uint64))
    short = full & ~np.uint64((1 << 30) - 1)
    return np.choose(rng.integers(0, 4, n), [full, ones, sparse, short])


def _values(rng, n, lo, hi):
    e = rng.integers(1023 + lo, 1023 + hi + 1, n).astype(np.uint64)
    s = rng.integers(0, 2, n).astype(np.uint64)
    return ((s << np.uint64(63)) | (e << np.uint64(52)) | _mantissas(rng, n)).view(np.float64)


def _special(rng, x):
    """Zeros, infinities, NaNs and denormals among x."""
    pick = rng.integers(0, 64, x.size)
    for k, v in enumerate((0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -3e-310, 1.0, 2.0 ** -700, 2.0 ** -701)):
        x[pick == k] = v
    return x


def _ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def _same(a, b):
    return a.view(np.uint64) == b.view(np.uint64)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["near_one", "in_range", "beyond", "special"])
def test_quotients_are_the_operators(lib, kind):
    rng = np.random.default_rng(11)
    n = 1 << 21
    ra, rb = {"near_one": ((-2, 2), (-2, 2)), "in_range": ((-699, 299), (-199, 199)),
              "beyond": ((-1021, 1022), (-1021, 1022)), "special": ((-720, 310), (-210, 210))}[kind]
    a, b = _values(rng, n, *ra), _values(rng, n, *rb)
    if kind == "special":
        a, b = _special(rng, a), _special(rng, b)
    q, q0, inv = (np.empty(n) for _ in range(3))
    ok = np.empty(n, np.int32)
    assert lib.run_quots(_ptr(a), _ptr(b), ctypes.c_long(n), _ptr(q), _ptr(q0), _ptr(inv), _ptr(ok)) == 0
    with np.errstate(all="ignore"):
        want, winv = a / b, 1.0 / b
    for got, w, bit in ((q, want, 1), (q0, want, 2), (inv, winv, 4)):
        took = (ok & bit) != 0
        bad = took & ~_same(got, w)
        assert not bad.any(), (kind, bit, a[bad][:3], b[bad][:3], got[bad][:3], w[bad][:3])
    if kind in ("near_one", "in_range"):
        assert (ok == 7).all()
    zero = (a == 0) & ((ok & 4) != 0)
    assert ((ok[zero] & 2) != 0).all() and ((ok[zero] & 1) == 0).all()


def _quotient_hard_cases(n, most):
    """a, b with a / b = N / 2^53 (1 + c / (b N)), N odd of 54 bits and |c| <= most odd: c / b ulp halves
    from the midpoint N / 2 of two doubles, where 1 / b is the nearest that a quotient can come."""
    rng = np.random.default_rng(13)
    a, b = [], []
    while len(a) < n:
        d = int(rng.integers(1 << 51, 1 << 52)) * 2 + 1   # an odd divisor of 53 bits
        c = int(rng.integers(0, most + 1)) // 2 * 2 + 1
        c = c if rng.integers(0, 2) else -c
        N = (-c * pow(d, -1, 1 << 54)) % (1 << 54)
        if N >= 1 << 53:
            a.append((d * N + c) >> 54)
            b.append(d)
    return a, b


def test_quotient_hard_cases_are_found():
    for a, b in zip(*_quotient_hard_cases(200, 63)):
        assert a < 1 << 53 and b < 1 << 53
        r = (a << 54) % b   # of 2 (a / b) in units of the quotient's half ulp
        assert min(r, b - r) <= 63 and round((a << 54) / b) >= 1 << 53


@pytest.mark.gpu
@pytest.mark.parametrize("most", [1, 63, 4095])
def test_quotients_next_to_midpoints(lib, most):
    ia, ib = _quotient_hard_cases(100000, most)
    a, b = np.array(ia, dtype=np.float64), np.array(ib, dtype=np.float64)
    rng = np.random.default_rng(14)
    s = rng.integers(-150, 150, a.size)   # anywhere in the divisors' range
    a = np.ldexp(a * rng.choice([-1.0, 1.0], a.size), rng.integers(-600, 200, a.size))
    b = np.ldexp(b, s - 52)
    n = a.size
    q, q0, inv = (np.empty(n) for _ in range(3))
    ok = np.empty(n, np.int32)
    assert lib.run_quots(_ptr(a), _ptr(b), ctypes.c_long(n), _ptr(q), _ptr(q0), _ptr(inv), _ptr(ok)) == 0
    assert (ok == 7).all()
    assert _same(q, a / b).all() and _same(q0, a / b).all() and _same(inv, 1.0 / b).all()


@pytest.mark.gpu
def test_the_approximations_at_every_mantissa(lib):
    """Both read a double's high word; |1 - b y| < 2^-19.9 and |1 - x z^2| < 2^-19.0 hold over all low words if
    they hold at the ends, as y and z are the same for all and the products are monotonic."""
    hi = np.arange(1 << 21, dtype=np.uint64) + np.uint64(1023 << 20)   # [1, 4): both parities of the exponent
    lo = [hi << np.uint64(32), (hi << np.uint64(32)) | np.uint64(0xffffffff)]
    lo.append((hi << np.uint64(32)) | np.random.default_rng(15).integers(0, 1 << 32, hi.size, dtype=np.uint64))
    got = []
    for bits in lo:
        x = bits.view(np.float64)
        y, z, ok = np.empty(x.size), np.empty(x.size), np.empty(x.size, np.int32)
        assert lib.run_starts(_ptr(x), ctypes.c_long(x.size), _ptr(y), _ptr(z), _ptr(ok)) == 0
        got.append((x.astype(np.longdouble), y.astype(np.longdouble), z.astype(np.longdouble)))
    for x, y, z in got:   # 21 significant bits in y and z: the products are exact to 2^-63
        assert (y == got[0][1]).all() and (z == got[0][2]).all()
        assert np.abs(1 - x * y).max() < 2.0 ** -19.9
        assert np.abs(1 - x * z * z).max() < 2.0 ** -19.0


def _root_hard_cases(most):
    """x in [1, 4) with 4 x 2^104 - M^2 = c for an odd M in [2^53, 2^54) and |c| <= most."""
    out = []
    for c in range(-most, most + 1):
        if (-c) % 8 != 1:
            continue
        for k in (54, 55):
            roots = [1, 3, 5, 7]
            for j in range(3, k):   # roots of M^2 = -c modulo 2^(j+1) from those modulo 2^j
                roots = sorted({r + d for r in roots for d in (0, 1 << (j - 1), 1 << j) if ((r + d) ** 2 + c) % (1 << (j + 1)) == 0 and r + d < 1 << (j + 1)})
            for r in roots:
                for m in range(r, 1 << 54, 1 << k):
                    x = (m * m + c) // 4
                    if m >= 1 << 53 and (x >> 104) in (1, 2, 3) and x % (1 << (52 if x < 1 << 105 else 53)) == 0:
                        out.append(float(x) / 2.0 ** 104)
    return np.array(sorted(set(out)))


def test_root_hard_cases_are_found():
    x = _root_hard_cases(64)
    assert x.size >= 16   # 16 values of c, about 1.4 x for each
    for v in x:
        n = int(v * 2.0 ** 52) << 52
        m = math.isqrt(4 * n)
        assert min(abs(4 * n - (m + d) ** 2) for d in (0, 1) if (m + d) % 2) <= 64


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["hard", "near_one", "in_range", "beyond", "special"])
def test_roots_are_the_library_s(lib, kind):
    rng = np.random.default_rng(12)
    n = 1 << 21
    if kind == "hard":
        base = _root_hard_cases(2048)
        x = np.concatenate([base * 2.0 ** e for e in (-850, -398, -2, 0, 2, 396)])
        n = x.size
    else:
        lo, hi = {"near_one": (-1, 1), "in_range": (-849, 398), "beyond": (-1021, 1022), "special": (-860, 410)}[kind]
        x = _values(rng, n, lo, hi)
        if kind in ("near_one", "in_range"):
            x = np.abs(x)
        if kind == "special":
            x = _special(rng, x)
    x = np.ascontiguousarray(x)
    r = np.empty(n)
    ok = np.empty(n, np.int32)
    assert lib.run_roots(_ptr(x), ctypes.c_long(n), _ptr(r), _ptr(ok)) == 0
    with np.errstate(all="ignore"):
        want = np.sqrt(x)
        assert (ok[x < 0] == 0).all()
    bad = (ok != 0) & ~_same(r, want)
    assert not bad.any(), (kind, x[bad][:3], r[bad][:3], want[bad][:3])
    if kind in ("hard", "near_one", "in_range"):
        assert ok.all()
