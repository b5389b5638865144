"""Batched contexts of different sizes alive at once: a kernel's shared-memory limit belongs to the process, so a later
context with smaller groups must not take away what an earlier one needs."""
import numpy as np
import pytest

from dpgsolver_gb300.host.mixed import mixed_euler
from dpgsolver_gb300.host.mixed_types import mixed_tri_quad_euler, mixed_types_euler

pytestmark = pytest.mark.gpu

MESHES = {
    "types": (lambda: mixed_types_euler(4, p_set=(1, 2, 3, 4), seed=0), lambda: mixed_types_euler(4, p_set=(1,), seed=0)),
    "types_p4_first": (lambda: mixed_types_euler(4, p_set=(4,), seed=0), lambda: mixed_types_euler(4, p_set=(2,), seed=0)),
    "tri_quad": (lambda: mixed_tri_quad_euler(6, p_set=(1, 4), seed=0), lambda: mixed_tri_quad_euler(6, p_set=(2,), seed=0)),
    "orders": (lambda: mixed_euler(3, 4, p_set=(1, 2, 3, 4)), lambda: mixed_euler(3, 4, p_set=(4,))),
}


@pytest.mark.parametrize("name", sorted(MESHES))
@pytest.mark.parametrize("form", ["plain", "fused", "branches", "stage"])
def test_a_smaller_context_leaves_the_larger_one_usable(gpu_lib, name, form):
    from dpgsolver_gb300.solver import BatchSimulation
    large, small = (make() for make in MESHES[name])
    with BatchSimulation(large) as a:
        a.form = form
        a.compute_rhs()
        r = a.rhs
        with BatchSimulation(small) as b:
            b.form = form
            b.compute_rhs()
            a.compute_rhs()
            assert np.array_equal(a.rhs, r)
            a.ssp_rk3_steps(large.dt, 1)
            b.ssp_rk3_steps(small.dt, 1)
        assert np.all(np.isfinite(a.sol_coef))
