"""Boundary states of the Euler equations at any scale: density scaled by 2^a and velocity by 2^b (pressure and energy by
2^(a + 2b), temperature by 2^2b), in the state and in the boundaries' data, scale the residual exactly. The tolerance is
the 1e-12 of the other parity tests."""
import numpy as np
import pytest

import oracle
from dpgsolver_gb300.host import problem as P

pytestmark = pytest.mark.gpu

CASES = {
    "riemann2d": lambda: P.euler_riemann_2d(5, 3),
    "channel2d": lambda: P.euler_channel_2d(4, 2),
    "duct3d": lambda: P.euler_duct_3d(3, 2),
    "subduct2d": lambda: P.euler_subsonic_duct(2, 4, 3),
    "subduct3d": lambda: P.euler_subsonic_duct(3, 3, 2),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("a,b", [(0, 0), (40, 0), (-40, 20), (300, 0), (-300, 0), (200, -100), (-150, 100)])
def test_scaled_boundary_states(gpu_lib, name, a, b):
    from dpgsolver_gb300.solver import Simulation
    prob = CASES[name]()
    ref, _ = oracle.Oracle(prob).compute_rhs(prob.sol)
    k = np.array([a] + [a + b] * prob.d + [a + 2 * b])
    prob.bc_state = np.ldexp(prob.bc_state, k)
    if prob.bc_data is not None:
        p_back, t_total, p_total, r_s = prob.bc_data
        prob.bc_data = (p_back * 2.0 ** (a + 2 * b), t_total * 2.0 ** (2 * b), p_total * 2.0 ** (a + 2 * b), r_s)
    with Simulation(prob) as sim:
        sim.upload_state(np.ldexp(prob.sol, k[None, :, None]))
        sim.compute_rhs()
        r = np.ldexp(sim.rhs, -(k + b)[None, :, None])
    assert np.max(np.abs(r - ref)) <= 1e-12 * np.max(np.abs(ref))
