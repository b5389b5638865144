"""The entries of the assembled Jacobian one by one, against the oracle evaluated in extended precision.

An entry far from its column's node is a small sum of products, and keeps the relative precision that FP64 arithmetic gives
it: the bar is the oracle's own FP64 evaluation (dense operators, complex step). The extended evaluation is the same
source compiled for long double complex (64 bits of mantissa or more) with a step of 1e-40, up to M^-1, which is applied
here in long double."""
import importlib.util
import os
import subprocess

import numpy as np
import pytest

import oracle
from dpgsolver_gb300.host import problem as P
from dpgsolver_gb300.host.problem import flat_arrays

pytestmark = pytest.mark.gpu
L = np.longdouble


@pytest.fixture(scope="module")
def extended(tmp_path_factory):
    """The oracle module on a library whose complex instantiation is long double and stops before M^-1; its results come as
    a double and the rest."""
    here, out = os.path.dirname(oracle.__file__), tmp_path_factory.mktemp("extended")
    with open(os.path.join(here, "dg_oracle.c")) as fh:
        src = fh.read()
    for a, b in (("double complex", "long double complex"), ("creal(x)", "creall(x)"), ("cabs(x)", "cabsl(x)"),
                 ("csqrt(x)", "csqrtl(x)"), ("cpow(x, y)", "cpowl(x, y)"), ("scale_m_inv_c(c, r);", ""),
                 ("s[i] = sol_re[i] + I * (sol_im ? sol_im[i] : 0.0);",
                  "s[i] = (long double)sol_re[i] + I * 1e-40L * (long double)sol_im[i];"),
                 ("rhs_re[i] = creal(r[i]);", "rhs_re[i] = (double)(cimagl(r[i]) * 1e40L);"),
                 ("rhs_im[i] = cimag(r[i]);", "rhs_im[i] = (double)(cimagl(r[i]) * 1e40L - rhs_re[i]);")):
        assert a in src
        src = src.replace(a, b)
    (out / "dg_oracle.c").write_text(src)
    so = str(out / "liboracle.so")
    subprocess.run(["gcc", "-O2", "-std=c11", "-fPIC", "-ffp-contract=off", "-I", here, "-shared", "-o", so,
                    str(out / "dg_oracle.c"), "-lm"], check=True)
    spec = importlib.util.spec_from_file_location("oracle_extended", oracle.__file__)
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    mod._LIB_PATH, mod._stale = so, lambda: False
    return mod


def _m_inv(prob):
    V = prob.ops.cv0_vs_vc().astype(L)
    X, eye = np.linalg.inv(V.astype(float)).astype(L), np.eye(len(V), dtype=L)
    for _ in range(3):
        X = X @ (2 * eye - V @ X)
    wJ = prob.ops.w_vc.astype(L) * np.reshape(flat_arrays(prob)["jacobian_det_vc"], (prob.n_volumes, 1, -1)).astype(L)
    return lambda raw: ((raw @ X) / wJ) @ X.T


@pytest.mark.parametrize("p", [2, 3])
def test_entries_as_precise_as_fp64(gpu_lib, extended, p):
    from dpgsolver_gb300.solver import Simulation
    prob = P.euler_hex_3d(3, p, num_flux=P.NUM_FLUX_LAX_FRIEDRICHS)
    u = prob.sol.copy()
    u[:, 0] *= 1.0 + 1e-2 * np.random.default_rng(3).uniform(-1, 1, u[:, 0].shape)
    with Simulation(prob) as sim:
        row_ptr, col_idx, vals = sim.jacobian(u, raw=False)
    w, minv = 13, _m_inv(prob)
    ext, fp64 = extended.Oracle(prob), oracle.Oracle(prob)
    blocks = [(v, b) for v in range(prob.n_volumes) for b in range(row_ptr[v], row_ptr[v + 1]) if col_idx[b] == w]
    got, ref, dense = [], [], []
    n = u[w].size
    for k in range(0, n, n // 10):
        e = np.zeros_like(u)
        e[w].reshape(-1)[k] = 1.0
        hi, lo = ext.compute_rhs_cmplx(u, e)
        x = minv(hi.astype(L) + lo.astype(L)).reshape(prob.n_volumes, -1)
        y = fp64.compute_rhs_cmplx(u, 1e-30 * e)[1].reshape(prob.n_volumes, -1) / 1e-30
        for v, b in blocks:
            got.append(vals[b][:, k])
            ref.append(x[v])
            dense.append(y[v])
    got, ref, dense = np.concatenate(got), np.concatenate(ref), np.concatenate(dense)
    m = np.abs(ref) > 1e-6 * np.max(np.abs(ref))
    for q in (0.5, 0.9):
        err = [float(np.quantile((np.abs(a - ref)[m] / np.abs(ref[m])).astype(float), q)) for a in (got, dense)]
        assert err[0] <= err[1], (q, err)
