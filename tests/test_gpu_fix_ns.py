"""The Navier-Stokes kernels on states that their fixed-point contractions do not take (non-finite values, a density spread,
magnitudes out of range): such an element's FP64 loops against the CPU oracle. Tolerances as in test_gpu_ns.py (1e-12 or
the oracle's noise), for a spread density times the largest ratio by which the flux divides."""
import numpy as np
import pytest

import oracle
from dpgsolver_gb300.host import problem as P
from test_gpu_ns import noise_floor, rel

pytestmark = pytest.mark.gpu


def _prob(d, p, flux=P.NUM_FLUX_ROE_PIKE):
    return P.ns_vortex_2d(4, p, num_flux=flux) if d == 2 else P.ns_taylor_green(3, p, Re=100.0, mach=0.3, num_flux=flux)


def _rhs(prob, sol):
    from dpgsolver_gb300.solver import Simulation
    with Simulation(prob) as sim:
        sim.upload_state(sol)
        sim.compute_rhs()
        return sim.rhs


@pytest.mark.parametrize("d,p", [(2, 1), (2, 4), (3, 2), (3, 3)])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_values(gpu_lib, d, p, bad):
    """They reach the elements that the dense operators carry them to, and no other element changes a bit."""
    prob = _prob(d, p)
    r0 = _rhs(prob, prob.sol)
    sol = prob.sol.copy()
    sol[5, 0, 1] = bad
    with np.errstate(all="ignore"):
        ref, _ = oracle.Oracle(prob).compute_rhs(sol)
    r = _rhs(prob, sol)
    hit = np.any(~np.isfinite(ref), axis=(1, 2))
    assert 1 <= hit.sum() < prob.n_volumes
    assert np.array_equal(np.any(~np.isfinite(r), axis=(1, 2)), hit)
    assert np.array_equal(r[~hit], r0[~hit])


@pytest.mark.parametrize("d,p", [(2, 1), (2, 3), (3, 2), (3, 4)])
@pytest.mark.parametrize("scale", [2.0 ** -3, 2.0 ** -12, 1e-9])
def test_density_spread(gpu_lib, d, p, scale):
    """One node at a fraction of its density, velocity and pressure kept: on either side of the spread rule."""
    prob = _prob(d, p)
    sol = prob.sol.copy()
    n = prob.ops.n_vs // 2
    ke = 0.5 * np.sum(sol[4, 1:1 + d, n] ** 2) / sol[4, 0, n]
    sol[4, :1 + d, n] *= scale
    sol[4, 1 + d, n] += (scale - 1.0) * ke
    ref, _ = oracle.Oracle(prob).compute_rhs(sol)
    r = _rhs(prob, sol)
    ok = np.isfinite(ref)
    assert np.array_equal(np.isfinite(r), ok)
    # the viscous flux divides by the density twice
    assert np.max(np.abs(np.where(ok, r - ref, 0.0))) <= 1e-12 * max(1.0, (1e-2 / scale) ** 2) * np.max(np.abs(ref[ok]))


@pytest.mark.parametrize("flux", [P.NUM_FLUX_ROE_PIKE, P.NUM_FLUX_LAX_FRIEDRICHS])
@pytest.mark.parametrize("d,p", [(2, 2), (3, 3)])
@pytest.mark.parametrize("a", [-400, -61, 0, 61, 400])
def test_scaled_density(gpu_lib, flux, d, p, a):
    """Density, pressure and viscosity scaled by 2^a scale the residual exactly, inside and beyond the range of
    the integer products (far beyond it the square of 1 / density leaves the exponent range)."""
    prob = _prob(d, p, flux)
    o = oracle.Oracle(prob)
    ref, _ = o.compute_rhs(prob.sol)
    tol = max(1e-12, 4.0 * noise_floor(o, prob.sol, ref))
    prob.ns = dict(prob.ns, mu=float(np.ldexp(prob.ns["mu"], a)))
    r = np.ldexp(_rhs(prob, np.ldexp(prob.sol, a)), -a)
    assert rel(r, ref) <= tol
