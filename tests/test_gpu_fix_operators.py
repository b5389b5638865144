"""Operators that have no fixed-point form (csrc/dgpu_host_ops.h, fix_usable): their elements stay in FP64 arithmetic, which
carries a NaN on and takes a basis of any scale. A residual in a basis scaled by powers of two is the scaled residual; the
tolerance is the 1e-12 of the other parity tests."""
import numpy as np
import pytest

import oracle
from dpgsolver_gb300.host import problem as P
from dpgsolver_gb300.host.mixed_types import mixed_tri_quad_euler, mixed_types_euler
from dpgsolver_gb300.host.simplex import WEDGE

pytestmark = pytest.mark.gpu


def _rhs(prob, sol):
    from dpgsolver_gb300.solver import BatchSimulation, Simulation
    with (BatchSimulation if hasattr(prob, "groups") else Simulation)(prob) as sim:
        sim.upload_state(sol)
        sim.compute_rhs()
        return sim.rhs


def _uniform(name, p):
    return {"advection": lambda: P.advection_2d(4, p), "euler2": lambda: P.euler_vortex_2d(4, p),
            "euler3": lambda: P.euler_hex_3d(2, p)}[name]()


@pytest.mark.parametrize("name,p", [("advection", 2), ("euler2", 1), ("euler2", 4), ("euler3", 2), ("euler3", 3)])
@pytest.mark.parametrize("op", ["cv1_1d", "cv0_bnd_1d"])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_operator_of_tensor_product_volumes(gpu_lib, name, p, op, bad):
    """One entry reaches every volume (it is a NaN or Inf in each sum of its row of Dgl or of the traces)."""
    prob = _uniform(name, p)
    a = np.array(getattr(prob.ops, op))
    a[0, 1] = bad
    setattr(prob.ops, op, a)
    with np.errstate(all="ignore"):
        r = _rhs(prob, prob.sol)
    assert np.all(np.any(~np.isfinite(r), axis=(1, 2)))


@pytest.mark.parametrize("kind", ["types", "tri_quad"])
@pytest.mark.parametrize("op", ["cv1_vs_vc", "cv0_vs_fc"])
def test_nan_operator_of_dense_volumes(gpu_lib, kind, op):
    make = {"types": lambda: mixed_types_euler(4, p_set=(1, 2), seed=0),
            "tri_quad": lambda: mixed_tri_quad_euler(6, p_set=(1, 3), seed=0)}[kind]
    n_dense = 0
    for g in range(len(make().groups)):
        prob = make()
        ops = prob.groups[g]
        if not getattr(ops, "dense", False) or not len(prob.group_vols[g]):
            continue
        if ops.e_type == WEDGE and op == "cv1_vs_vc":
            ops.prism_factors = _nan_factors(ops.prism_factors())
        n_dense += 1
        f = getattr(ops, op)

        def bad(*a, f=f):
            x = np.array(f(*a))
            x[0, 0] = np.nan
            return x
        setattr(ops, op, bad)
        try:
            r = _rhs(prob, prob.sol)
        except Exception as e:   # factors that do not reproduce the dense operators are refused
            assert "WEDGE factors" in str(e)
            continue
        off = prob.state_off
        for v in prob.group_vols[g]:
            assert not np.all(np.isfinite(r[off[v]:off[v + 1]]))
    assert n_dense >= 2


def _nan_factors(factors):
    t0, t1, l0, l1 = (np.array(x) for x in factors)
    t1.reshape(-1)[0] = np.nan
    return lambda: (t0, t1, l0, l1)


@pytest.mark.parametrize("name,p", [("advection", 2), ("euler2", 3), ("euler3", 2), ("euler3", 4)])
@pytest.mark.parametrize("scale", [2, 30, 110, -40, "uneven"])
def test_scaled_nodal_basis(gpu_lib, name, p, scale):
    prob = _uniform(name, p)
    ref, _ = oracle.Oracle(prob).compute_rhs(prob.sol)
    q, d = p + 1, prob.d
    s = np.ldexp(1.0, scale) * np.ones(q) if scale != "uneven" else np.ldexp(1.0, 40 * (np.arange(q) == 1))
    for op in ("cv0_1d", "cv1_1d", "cv0_bnd_1d"):
        setattr(prob.ops, op, getattr(prob.ops, op) * s)
    prob.ops.ccSB0_1d, prob.ops.ccBS0_1d = prob.ops.ccSB0_1d * s, prob.ops.ccBS0_1d / s[:, None]
    f = s
    for _ in range(d - 1):
        f = np.multiply.outer(s, f).reshape(-1)
    r = _rhs(prob, prob.sol / f) * f
    assert np.max(np.abs(r - ref)) <= 1e-12 * np.max(np.abs(ref))


@pytest.mark.parametrize("kind", ["types", "tri_quad"])
@pytest.mark.parametrize("scale", [2, 30, 110, -40, "uneven"])
def test_scaled_dense_basis(gpu_lib, kind, scale):
    prob = mixed_types_euler(4, p_set=(1, 2, 3), seed=0) if kind == "types" else \
        mixed_tri_quad_euler(6, p_set=(1, 2, 4), seed=0)
    ref, _ = oracle.Oracle(prob).compute_rhs(prob.sol)
    sol, back = prob.sol.copy(), np.ones_like(prob.sol)
    for g, ops in enumerate(prob.groups):
        if not getattr(ops, "dense", False) or not len(prob.group_vols[g]):
            continue
        n = np.arange(ops.n_vs)
        if ops.e_type == WEDGE:   # the TRI factor's functions, on every one of the LINE's
            n = n % ops.prism_factors()[0].shape[1]
        s = np.ldexp(1.0, 40 * (n == 1)) if scale == "uneven" else np.ldexp(1.0, scale) * np.ones(ops.n_vs)
        for op in ("cv0_vs_vc", "cv1_vs_vc", "cv0_vs_fc", "ccSB0_vs_vs"):
            setattr(ops, op, lambda *a, f=getattr(ops, op), s=s: f(*a) * s)
        setattr(ops, "ccBS0_vs_vs", lambda f=ops.ccBS0_vs_vs, s=s: f() / s[:, None])
        if ops.e_type == WEDGE:
            setattr(ops, "prism_factors", lambda f=ops.prism_factors(), s=s[:max(n) + 1]: (f[0] * s, f[1] * s, f[2], f[3]))
        prob.set_group(sol, g, prob.group_view(sol, g) / s)
        prob.set_group(back, g, prob.group_view(back, g) * s)
    r = _rhs(prob, sol) * back
    assert np.max(np.abs(r - ref)) <= 1e-12 * np.max(np.abs(ref))

