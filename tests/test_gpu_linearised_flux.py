"""The linearised residual where its kernels branch: flow below, near and above the speed of sound in both directions (the
wave-speed branches of the fluxes' reverse mode), and tangents and cotangents at the ends of the block fixed-point range.

Both products are exact to rounding, so the bars are the 1e-12 of the other linearisation tests: of |v| |J d| for the
transpose, and of the largest value for the scaling, which is exact but for denormal results.
"""
import numpy as np
import pytest

import oracle
from dpgsolver_gb300.host import problem as P

pytestmark = pytest.mark.gpu


def _inputs(prob, mach):
    d = prob.d
    rng = np.random.default_rng(5)
    u = prob.sol + 1e-2 * rng.standard_normal(prob.sol.shape)
    rho, V = u[:, 0], u[:, 1:1 + d] / u[:, :1]
    p = 0.4 * (u[:, d + 1] - 0.5 * rho * np.sum(V * V, axis=1))
    V = V + (mach * np.sqrt(1.4 * np.max(p / rho)) * np.array([1.0, -0.6, 0.3])[:d])[None, :, None]
    u[:, 1:1 + d] = rho[:, None] * V
    u[:, d + 1] = p / 0.4 + 0.5 * rho * np.sum(V * V, axis=1)
    return u, rng.standard_normal(u.shape), rng.standard_normal(u.shape)


@pytest.mark.parametrize("flux", [P.NUM_FLUX_ROE_PIKE, P.NUM_FLUX_LAX_FRIEDRICHS])
@pytest.mark.parametrize("d,p", [(2, 1), (2, 4), (3, 1), (3, 2), (3, 4)])
@pytest.mark.parametrize("mach", [-3.0, -0.8, 0.4, 1.1, 5.0])
def test_products_against_complex_step(gpu_lib, flux, d, p, mach):
    from dpgsolver_gb300.solver import Simulation
    prob = P.euler_vortex_2d(4, p, num_flux=flux) if d == 2 else P.euler_hex_3d(2, p, num_flux=flux)
    u, dirn, v = _inputs(prob, mach)
    _, ri = oracle.Oracle(prob).compute_rhs_cmplx(u, 1e-30 * dirn)
    ref = ri / 1e-30
    with Simulation(prob) as sim:
        _, jv = sim.jvp(u, dirn)
        sim.vjp_forward(u)
        g = sim.vjp_backward(v)
    assert np.max(np.abs(jv - ref)) <= 1e-12 * np.max(np.abs(ref))
    assert abs(np.sum(g * dirn) - np.sum(v * ref)) <= 1e-12 * np.sqrt(np.sum(v * v) * np.sum(ref * ref))


@pytest.mark.parametrize("name", ["advection", "euler2", "euler3"])
@pytest.mark.parametrize("power", [-980, -830, -815, 815, 830, 980])
def test_scaled_tangent_and_cotangent(gpu_lib, name, power):
    from dpgsolver_gb300.solver import Simulation
    prob = {"advection": lambda: P.advection_2d(4, 3), "euler2": lambda: P.euler_vortex_2d(4, 2),
            "euler3": lambda: P.euler_hex_3d(2, 3)}[name]()
    rng = np.random.default_rng(6)
    u = prob.sol + 1e-2 * rng.standard_normal(prob.sol.shape)
    dirn, v = rng.standard_normal(u.shape), rng.standard_normal(u.shape)
    with Simulation(prob) as sim:
        _, j0 = sim.jvp(u, dirn)
        _, j1 = sim.jvp(u, np.ldexp(dirn, power))
        sim.vjp_forward(u)
        g0 = sim.vjp_backward(v)
        g1 = sim.vjp_backward(np.ldexp(v, power))
    for a, b in ((j0, j1), (g0, g1)):
        assert np.max(np.abs(np.ldexp(b, -power) - a)) <= 1e-12 * np.max(np.abs(a))
