"""Precision that FP64 arithmetic gives and block fixed point (csrc/dgpu_fix.cuh) would not: values far below their element's
largest one that nothing couples to it.

An advection velocity along x couples the nodes of a line along x to no other line, when the metric terms and normals of the
Cartesian mesh hold no rounding errors across it. For an odd number of nodes a direction
the middle line's nodes are nodes of both the solution and the cubature, so its residual depends on its own values
alone, however large the others are. FP64 sums of at most 5 terms are within 2^-50 of the sum of their terms' magnitudes;
three contractions, and the cancellation in the derivative, give the 1e-13 below."""
import numpy as np
import pytest

from dpgsolver_gb300.host import problem as P

pytestmark = pytest.mark.gpu


def _middle(prob):
    q = prob.ops.p + 1
    n = np.arange(q ** prob.d)
    return (n // q) % q == q // 2


def _exact(a):
    """Metric terms or normals of a Cartesian mesh: what is below rounding is zero."""
    return np.where(np.abs(a) < 1e-12 * np.max(np.abs(a)), 0.0, a)


def _states(prob, tiny):
    rng = np.random.default_rng(0)
    row = _middle(prob)
    u = rng.uniform(0.5, 1.0, prob.sol.shape)
    line = np.where(row, tiny * u, 0.0)
    return row, line, np.where(row, line, u)


@pytest.mark.parametrize("p", [2, 4])
@pytest.mark.parametrize("tiny", [1e-3, 1e-6, 1e-9, 1e-12])
@pytest.mark.parametrize("entry", ["rhs", "steps", "jvp"])
def test_decoupled_line_of_advection(gpu_lib, p, tiny, entry):
    from dpgsolver_gb300.solver import Simulation
    prob = P.advection_2d(4, p, b=(1.0, 0.0))
    prob.geom.metrics_vc, prob.geom.normals_fc = _exact(prob.geom.metrics_vc), _exact(prob.geom.normals_fc)
    row, line, full = _states(prob, tiny)

    def run(u):
        with Simulation(prob) as sim:
            if entry == "jvp":
                return sim.jvp(prob.sol, u)[1]
            sim.upload_state(u)
            if entry == "rhs":
                sim.compute_rhs()
                return sim.rhs
            sim.ssp_rk3_steps(prob.dt, 2)
            return sim.sol_coef
    alone, both = run(line)[:, :, row], run(full)[:, :, row]
    assert np.max(np.abs(both - alone)) <= 1e-13 * np.max(np.abs(alone))


@pytest.mark.parametrize("p_set", [(2,), (4,), (2, 4)])
@pytest.mark.parametrize("tiny", [1e-3, 1e-9])
def test_decoupled_line_of_batched_advection(gpu_lib, p_set, tiny):
    """As above; volumes of order 2 and 4 side by side interpolate their traces, which mixes the lines of a face, so there only
    the volumes whose neighbours in x have their own order are compared."""
    from dpgsolver_gb300.host.mixed import mixed_advection_2d
    from dpgsolver_gb300.solver import BatchSimulation
    prob = mixed_advection_2d(6, p_set=p_set, b=(1.0, 0.0))
    flat = prob.flat()
    flat["metrics_vc"], flat["normals_fc"] = _exact(flat["metrics_vc"]), _exact(flat["normals_fc"])
    prob.flat = lambda: flat
    rng = np.random.default_rng(1)
    line, full = np.zeros_like(prob.sol), prob.sol.copy()
    rows = []
    for g, ops in enumerate(prob.groups):
        q = ops.p + 1
        row = (np.arange(q * q) // q) % q == q // 2
        u = rng.uniform(0.5, 1.0, prob.group_view(full, g).shape)
        prob.set_group(line, g, np.where(row, tiny * u, 0.0))
        prob.set_group(full, g, np.where(row, tiny * u, u))
        rows.append(row)
    fv = prob.mesh.face_vol
    mixed = np.zeros(prob.n_volumes, dtype=bool)
    for a, b in fv[prob.vol_group[fv[:, 0]] != prob.vol_group[fv[:, 1]]]:
        mixed[[a, b]] = True

    def run(u):
        with BatchSimulation(prob) as sim:
            sim.upload_state(u)
            sim.compute_rhs()
            return sim.rhs
    a, b = run(line), run(full)
    for g, row in enumerate(rows):
        keep = ~mixed[prob.group_vols[g]]
        x, y = prob.group_view(a, g)[keep][:, :, row], prob.group_view(b, g)[keep][:, :, row]
        if x.size:
            assert np.max(np.abs(y - x)) <= 1e-13 * np.max(np.abs(x))
