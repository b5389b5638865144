"""The volume term's fixed-point contractions (csrc/dgpu_tp.cuh on csrc/dgpu_fix.cuh) value by value, in extended precision:
how far a density, an energy or a momentum may lie below its element's largest one.

FP64 sums of q products are within q 2^-53 of sum |w x|. A value is held to 3 2^-59 of its block's largest one, and the dropped
low products and the operators' own rounding come to 6 terms 2^-62 of that times sum |w| at most. With densities and
energies within 2^5 of each other in an element (the spread rule) this is below the FP64 bound of the density and energy of each
line, and for the momentum, at most sqrt(2 rho E) where the pressure is positive, below that of sqrt(2 rho E)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from dpgsolver_gb300 import _lib
from dpgsolver_gb300.host import problem as P

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
L = np.longdouble
U = 2.0 ** -53
SHAPES = [(2, 2), (2, 4), (3, 1), (3, 3)]


@pytest.fixture(scope="module")
def volume(gpu_lib, tmp_path_factory):
    so = str(tmp_path_factory.mktemp("probe") / "libfix_probe.so")
    subprocess.run([_lib.nvcc_path()] + _lib.NVCC_FLAGS + ["-shared", "-I", _lib.CSRC, "-o", so,
                                                           os.path.join(HERE, "cuda", "fix_probe.cu")], check=True)
    fn = ctypes.CDLL(so).fix_probe_volume
    dp, ip = _lib.c_double_p, _lib.c_int_p
    fn.argtypes = [ctypes.c_int, ctypes.c_int, dp, dp, dp, ctypes.c_int, dp, dp, dp, dp, ip, dp, dp]

    def run(d, p, W, F):
        ops = (P.advection_2d(3, p) if d == 2 else P.euler_hex_3d(2, p)).ops
        n, nv, N = W.shape
        q, nf = p + 1, N // (p + 1)
        a = [np.ascontiguousarray(x) for x in (ops.cv0_1d, ops.cv1_1d, ops.cv0_bnd_1d, W, F)]
        traces, vol, fixed = np.empty((n, 2 * d, nv, nf)), np.empty((n, nv, N)), np.empty(n, dtype=np.int32)
        lb, Dgl = np.empty((2, 5)), np.empty((5, 5))
        ptr = [x.ctypes.data_as(dp) for x in a + [traces, vol, lb, Dgl]]
        assert fn(d, p, *ptr[:3], n, ptr[3], ptr[4], ptr[5], ptr[6], fixed.ctypes.data_as(ip), ptr[7], ptr[8]) == 0
        return traces, vol, fixed, lb[:, :q], Dgl[:q, :q]
    return run


def _lines(d, q, x):
    """x (.., N) with the nodes of the lines along direction k last: k -> (.., lines, q)."""
    g = x.reshape(x.shape[:-1] + (q,) * d)
    return [np.moveaxis(g, -1 - k, -1).reshape(x.shape[:-1] + (q ** (d - 1), q)) for k in range(d)]


def _trace_ref(d, q, lb, x):
    """Traces of x (n, nv, N): (n, 2 d, nv, q^(d-1)), face 2 k + s."""
    return np.stack([ln @ lb[s].astype(L) for ln in _lines(d, q, x.astype(L)) for s in (0, 1)], axis=1)


def _state(rng, n, d, N):
    rho = rng.uniform(0.5, 1.0, (n, 1, N))
    vel = rng.uniform(-1.0, 1.0, (n, d, N))
    E = 2.5 * rng.uniform(0.5, 1.0, (n, 1, N)) + 0.5 * rho * np.sum(vel * vel, axis=1, keepdims=True)
    return np.concatenate([rho, rho * vel, E], axis=1)


@pytest.mark.parametrize("d,p", SHAPES)
@pytest.mark.parametrize("var", ["density", "energy"])
@pytest.mark.parametrize("k", [0, 2, 3, 5, 6, 8, 12, 40, 300])
def test_low_line_of_a_state(volume, d, p, var, k):
    """The density (or the energy, at rest) of one line of nodes 2^-k below the others': its trace to FP64's own bound, by the
    spread rule in fixed point or by the FP64 loops, which side is told for the k that leave no doubt."""
    q, n = p + 1, 13
    N, rng = q ** d, np.random.default_rng(k)
    W = _state(rng, n, d, N)
    low = np.arange(N) // q == 1
    if var == "density":
        W[:, :1 + d, low] *= 2.0 ** -k
    else:
        W[:, 1:, low] *= 2.0 ** -k
    F = rng.uniform(-1.0, 1.0, (n, d, d + 2, N))
    traces, _, fixed, lb, _ = volume(d, p, W, F)
    if k <= 2:
        assert np.all(fixed == 1)
    if k >= 6:
        assert np.all(fixed == 0)
    ref, mag = _trace_ref(d, q, lb, W), _trace_ref(d, q, np.abs(lb), np.abs(W))
    for m in (0, d + 1):
        assert np.all(np.abs(traces[:, :, m] - ref[:, :, m]) <= q * U * mag[:, :, m])


@pytest.mark.parametrize("d,p", SHAPES)
@pytest.mark.parametrize("k", [0, 10, 30, 60, 200])
def test_low_momentum(volume, d, p, k):
    """Momentum of one line 2^-k below the others': to FP64's bound of sqrt(2 rho E), the scale of what a flux adds it to."""
    q, n = p + 1, 13
    N, rng = q ** d, np.random.default_rng(100 + k)
    W = _state(rng, n, d, N)
    W[:, 1:1 + d, np.arange(N) // q == 1] *= 2.0 ** -k
    F = rng.uniform(-1.0, 1.0, (n, d, d + 2, N))
    traces, _, fixed, lb, _ = volume(d, p, W, F)
    ref = _trace_ref(d, q, lb, W)
    mag = _trace_ref(d, q, np.abs(lb), np.sqrt(2 * W[:, :1] * W[:, -1:]))
    assert np.all(np.abs(traces - ref)[:, :, 1:1 + d] <= q * U * mag)


@pytest.mark.parametrize("d,p", SHAPES)
@pytest.mark.parametrize("scale", [-700, 0, 700])
def test_derivative_within_the_stated_bound(volume, d, p, scale):
    """sum_j Dgl_j^T f_j of fluxes of very different sizes: within (3 2^-59 + 6 terms 2^-62) B sum |w| and its one rounding."""
    q, n = p + 1, 29
    N, rng = q ** d, np.random.default_rng(7)
    W = _state(rng, n, d, N)
    F = rng.choice([-1.0, 1.0], (n, d, d + 2, N)) * np.exp2(rng.uniform(-40.0, 0.0, (n, d, d + 2, N)))
    F = np.ldexp(F, scale)
    _, vol, fixed, _, D = volume(d, p, W, F)
    assert np.all(fixed == 1)
    ref, mag = np.zeros(vol.shape, dtype=L), np.zeros(vol.shape, dtype=L)
    g = np.zeros(N, dtype=L)
    for j in range(d):
        x = np.moveaxis(F[:, j].astype(L).reshape((n, d + 2) + (q,) * d), -1 - j, -1) @ D.astype(L)
        ref += np.moveaxis(x, -1, -1 - j).reshape(vol.shape)
        w = np.moveaxis(np.ones((q,) * d, dtype=L), -1 - j, -1) @ np.abs(D).astype(L)
        g += np.moveaxis(w, -1, -1 - j).reshape(N)
    B = np.exp2(np.floor(np.log2(np.max(np.abs(F), axis=(1, 3)))) + 1)[:, :, None]
    mag = B.astype(L) * np.max(g)
    bound = (3 * 2.0 ** -59 + 6 * d * q * 2.0 ** -62) * mag + U * np.abs(ref)
    assert np.all(np.abs(vol - ref) <= bound)
