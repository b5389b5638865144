"""Dense groups up to the largest volume cubature one CTA's shared memory takes: the rule's nodes repeated, their weights
shared out, which leaves the residual what it is (to the 1e-12 of the other parity tests)."""
import numpy as np
import pytest

import oracle
from dpgsolver_gb300 import _lib
from dpgsolver_gb300.host.mixed_types import mixed_types_euler
from dpgsolver_gb300.host.simplex import TET

pytestmark = pytest.mark.gpu


def _with_nodes(n_vc):
    """TET p1: 5 x 4 coefficients and 3 x 5 n_vc flux values a volume, at most 25,600 doubles."""
    prob = mixed_types_euler(4, p_set=(1,), seed=0)
    ref, _ = oracle.Oracle(prob).compute_rhs(prob.sol)
    ops = next(o for o in prob.groups if o.e_type == TET)
    at = np.resize(np.arange(ops.n_vc), n_vc)
    w = ops.w_vc[at] / np.bincount(at)[at]
    cv0, cv1 = ops.cv0_vs_vc()[at], [ops.cv1_vs_vc(k)[at] for k in range(3)]
    ops.n_vc, ops.w_vc, ops.cv0_vs_vc, ops.cv1_vs_vc = n_vc, w, lambda: cv0, lambda k: cv1[k]
    return prob, ref


@pytest.mark.parametrize("n_vc", [64, 800, 1704, 1705])
def test_long_cubature(gpu_lib, n_vc):
    from dpgsolver_gb300.solver import BatchSimulation
    prob, ref = _with_nodes(n_vc)
    with BatchSimulation(prob) as sim:
        for form in ("plain", "fused"):
            sim.form = form
            sim.compute_rhs()
            assert np.max(np.abs(sim.rhs - ref)) <= 1e-12 * np.max(np.abs(ref)), form


def test_longer_cubature_is_refused(gpu_lib):
    from dpgsolver_gb300.solver import BatchSimulation
    prob, _ = _with_nodes(1706)
    with pytest.raises(_lib.DGPUError, match="too large"):
        BatchSimulation(prob)
