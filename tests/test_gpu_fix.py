"""Block fixed-point contractions (csrc/dgpu_fix.cuh) at the edges of their range, against the CPU oracle.

The fixed-point sums are exact to a few 2^-59 of their largest term, below FP64's own rounding, so the tolerance is the
1e-12 of the other parity tests; a state outside the range takes the FP64 loops and meets the same tolerance.
"""
import numpy as np
import pytest

import oracle
from dpgsolver_gb300.host import problem as P

pytestmark = pytest.mark.gpu


def _residual(prob, sol):
    from dpgsolver_gb300.solver import Simulation
    with Simulation(prob) as sim:
        sim.upload_state(sol)
        back = sim.sol_coef
        sim.compute_rhs()
        return sim.rhs, back


@pytest.mark.parametrize("p", [1, 2, 3, 4])
@pytest.mark.parametrize("power", [-1000, -830, -818, 0, 818, 830, 990])
def test_scaled_advection(gpu_lib, p, power):
    """The linear residual scales exactly with the state, inside, at and beyond the ends of the block range."""
    prob = P.advection_2d(5, p)
    r0, _ = oracle.Oracle(prob).compute_rhs(prob.sol)
    r, back = _residual(prob, np.ldexp(prob.sol, power))
    assert np.array_equal(back, np.ldexp(prob.sol, power))
    r = np.ldexp(r, -power)
    assert np.max(np.abs(r - r0)) <= 1e-12 * np.max(np.abs(r0))


@pytest.mark.parametrize("d,p", [(2, 1), (2, 3), (3, 2), (3, 3), (3, 4)])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_values_stay_in_their_elements(gpu_lib, d, p, bad):
    """A NaN or Inf reaches the elements that the dense operators carry it to, and no other element changes a bit."""
    prob = P.euler_vortex_2d(5, p) if d == 2 else P.euler_hex_3d(4, p)
    r0, _ = _residual(prob, prob.sol)
    sol = prob.sol.copy()
    sol[7, 0, 1] = bad
    with np.errstate(all="ignore"):
        ref, _ = oracle.Oracle(prob).compute_rhs(sol)
    r, _ = _residual(prob, sol)
    hit = np.any(~np.isfinite(ref), axis=(1, 2))
    assert 1 <= hit.sum() < prob.n_volumes
    assert np.array_equal(np.any(~np.isfinite(r), axis=(1, 2)), hit)
    assert np.array_equal(r[~hit], r0[~hit])


@pytest.mark.parametrize("d,p", [(2, 2), (3, 2), (3, 3)])
@pytest.mark.parametrize("scale", [2.0 ** -3, 2.0 ** -12, 1e-9])
def test_density_spread(gpu_lib, d, p, scale):
    """One node of an element at a fraction of its density (velocity and pressure kept): the residual on either side of
    the spread rule."""
    prob = P.euler_vortex_2d(5, p) if d == 2 else P.euler_hex_3d(3, p)
    sol = prob.sol.copy()
    n = prob.ops.n_vs // 2
    sol[4, 0, n] *= scale
    sol[4, 1:1 + d, n] *= scale
    ref, _ = oracle.Oracle(prob).compute_rhs(sol)
    r, back = _residual(prob, sol)
    assert np.array_equal(back, sol)
    # the flux divides by densities down to scale: its rounding errors scale with the largest value at hand
    ok = np.isfinite(ref)
    assert np.array_equal(np.isfinite(r), ok)
    assert np.max(np.abs(np.where(ok, r - ref, 0.0))) <= 1e-12 * max(1.0, 1e-3 / scale) * np.max(np.abs(ref[ok]))


@pytest.mark.parametrize("flux", [P.NUM_FLUX_ROE_PIKE, P.NUM_FLUX_LAX_FRIEDRICHS])
@pytest.mark.parametrize("d", [2, 3])
@pytest.mark.parametrize("a,b", [(0, 0), (58, 0), (61, 0), (-58, 0), (-61, 0), (0, 29), (0, 31), (0, -29), (0, -90), (-200, 70)])
def test_scaled_euler(gpu_lib, flux, d, a, b):
    """Density scaled by 2^a and velocity by 2^b (momentum 2^(a+b), energy 2^(a+2b)): the residual scales exactly on
    either side of the range in which the fluxes use integer products."""
    prob = P.euler_vortex_2d(4, 2, num_flux=flux) if d == 2 else P.euler_hex_3d(3, 2, num_flux=flux)
    r0, _ = oracle.Oracle(prob).compute_rhs(prob.sol)
    k = np.array([a] + [a + b] * d + [a + 2 * b])[None, :, None]
    r, _ = _residual(prob, np.ldexp(prob.sol, k))
    r = np.ldexp(r, -k - b)
    assert np.max(np.abs(r - r0)) <= 1e-12 * np.max(np.abs(r0))


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("kind", ["types", "tri_quad"])
def test_non_finite_values_in_dense_groups(gpu_lib, bad, kind):
    """As test_non_finite_values_stay_in_their_elements, on meshes with dense groups, for one volume of every group."""
    from dpgsolver_gb300.host.mixed_types import mixed_tri_quad_euler, mixed_types_euler
    from dpgsolver_gb300.solver import BatchSimulation
    prob = mixed_types_euler(4, seed=0) if kind == "types" else mixed_tri_quad_euler(6, seed=0)
    o = oracle.Oracle(prob)
    with BatchSimulation(prob) as sim:
        sim.compute_rhs()
        r0 = sim.rhs
        for vols in prob.group_vols:
            if not len(vols):
                continue
            sol = prob.sol.copy()
            sol[prob.state_off[vols[0]]] = bad
            with np.errstate(all="ignore"):
                ref, _ = o.compute_rhs(sol)
            sim.upload_state(sol)
            sim.compute_rhs()
            r = sim.rhs
            off = prob.state_off
            hit = np.array([not np.all(np.isfinite(ref[off[v]:off[v + 1]])) for v in range(prob.n_volumes)])
            got = np.array([not np.all(np.isfinite(r[off[v]:off[v + 1]])) for v in range(prob.n_volumes)])
            assert hit.any() and np.array_equal(got, hit)
            same = np.repeat(~hit, np.diff(off))
            assert np.array_equal(r[same], r0[same])


@pytest.mark.parametrize("p", [1, 3, 4])
@pytest.mark.parametrize("power", [-1000, -900, 0, 900, 990])
def test_scaled_advection_steps(gpu_lib, p, power):
    """Two SSP-RK3 steps of the linear equation scale exactly with the state: the stage's products near both ends of the
    exponent range, where they go back to the FP64 pipe."""
    from dpgsolver_gb300.solver import Simulation
    prob = P.advection_2d(5, p)
    o = oracle.Oracle(prob)
    ref = prob.sol
    for _ in range(2):
        ref, _, _ = o.ssp_rk3_step(ref, prob.dt)
    with Simulation(prob) as sim:
        sim.upload_state(np.ldexp(prob.sol, power))
        sim.ssp_rk3_steps(prob.dt, 2)
        got = np.ldexp(sim.sol_coef, -power)
    assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))
