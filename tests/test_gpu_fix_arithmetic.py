"""The integer-pipe arithmetic of csrc/dgpu_fix.cuh against IEEE arithmetic, bit for bit."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from dpgsolver_gb300 import _lib

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
RCP, SQRT, DIV, MUL, MUL_INT = range(5)


@pytest.fixture(scope="module")
def probe(gpu_lib, tmp_path_factory):
    so = str(tmp_path_factory.mktemp("probe") / "libfix_probe.so")
    subprocess.run([_lib.nvcc_path()] + _lib.NVCC_FLAGS + ["-shared", "-I", _lib.CSRC, "-o", so,
                                                           os.path.join(HERE, "cuda", "fix_probe.cu")], check=True)
    fn = ctypes.CDLL(so).fix_probe
    fn.argtypes = [ctypes.c_int, _lib.c_double_p, _lib.c_double_p, _lib.c_double_p, ctypes.c_longlong]

    def run(op, a, b=None):
        a = np.ascontiguousarray(a)
        b = np.ascontiguousarray(np.broadcast_to(a if b is None else b, a.shape))
        out = np.empty_like(a)
        p = [x.ctypes.data_as(_lib.c_double_p) for x in (a, b, out)]
        assert fn(op, *p, a.size) == 0
        return out
    return run


def _same(got, ref):
    bad = (got.view(np.uint64) != ref.view(np.uint64)) & ~(np.isnan(got) & np.isnan(ref))
    assert not np.any(bad), (got[bad][:3], ref[bad][:3], int(bad.sum()))


def _random(rng, n, lo=1, hi=2046):
    e = rng.integers(lo, hi + 1, n, dtype=np.uint64) << np.uint64(52)
    m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    s = rng.integers(0, 2, n, dtype=np.uint64) << np.uint64(63)
    return (s | e | m).view(np.float64)


def _edges():
    """Every exponent with the mantissas next to a power of two and to the middle, both signs, and what is not normal."""
    m = np.array([0, 1, 2, 2 ** 51 - 1, 2 ** 51, 2 ** 51 + 1, 2 ** 52 - 2, 2 ** 52 - 1], dtype=np.uint64)
    x = ((np.arange(2048, dtype=np.uint64) << np.uint64(52))[:, None] | m).reshape(-1).view(np.float64)
    return np.concatenate([x, -x])


def test_every_leading_mantissa(probe):
    """The seeds are functions of the 23 leading bits: with each of them, the least, the largest and a random rest."""
    rng = np.random.default_rng(0)
    lead = (np.arange(1 << 23, dtype=np.uint64) << np.uint64(29))
    for e in (1022, 1023):
        for rest in (0, (1 << 29) - 1, rng.integers(0, 1 << 29, 1 << 23, dtype=np.uint64)):
            x = ((np.uint64(e) << np.uint64(52)) | lead | np.uint64(rest) if np.isscalar(rest)
                 else (np.uint64(e) << np.uint64(52)) | lead | rest).view(np.float64)
            _same(probe(RCP, x), 1.0 / x)
            _same(probe(SQRT, x), np.sqrt(x))
            a = _random(rng, x.size, 1000, 1050)
            _same(probe(DIV, a, x), a / x)


def test_exponent_edges(probe):
    x = _edges()
    with np.errstate(all="ignore"):
        _same(probe(RCP, x), 1.0 / x)
        _same(probe(SQRT, x), np.sqrt(x))
        for b in (1.0, -3.0, 0.1, 1e-300, 1.7e308, 2.0 ** -1022, 5e-324, 0.0, np.inf):
            _same(probe(DIV, x, b), x / b)
            _same(probe(DIV, np.full_like(x, b), x), b / x)
            _same(probe(MUL_INT, x, b), x * b)
            _same(probe(MUL_INT, np.full_like(x, b), x), b * x)


def test_random_arguments(probe):
    rng = np.random.default_rng(1)
    with np.errstate(all="ignore"):
        for _ in range(8):
            a, b = _random(rng, 1 << 22), _random(rng, 1 << 22)
            _same(probe(RCP, a), 1.0 / a)
            _same(probe(SQRT, np.abs(a)), np.sqrt(np.abs(a)))
            _same(probe(DIV, a, b), a / b)
            _same(probe(MUL_INT, a, b), a * b)


def test_products_in_range(probe):
    """fix_mul for zeros and normal factors with a normal product: random ones, ties to even and carries."""
    rng = np.random.default_rng(2)
    n = 1 << 21
    a, b = _random(rng, n, 600, 1400), _random(rng, n, 600, 1400)
    a[::101], b[::97] = 0.0, -0.0
    _same(probe(MUL, a, b), a * b)
    for k in (1, 2, 25, 26, 27, 51):   # short factors: exact products and exact halves of the last unit
        ai = rng.integers(1 << 52, 1 << 53, n, dtype=np.uint64)
        bi = (rng.integers(0, 1 << k, n, dtype=np.uint64) | np.uint64(1 << k))
        x, y = ai.astype(np.float64), bi.astype(np.float64)
        _same(probe(MUL, x, y), x * y)
        odd = (2 * rng.integers(1 << 51, 1 << 52, n, dtype=np.uint64) + 1).astype(np.float64)
        _same(probe(MUL, odd, np.full(n, 1.5)), odd * 1.5)
    one = np.nextafter(np.ldexp(1.0, np.arange(-300, 300)), 0.0)
    _same(probe(MUL, one, one[::-1].copy()), one * one[::-1])
