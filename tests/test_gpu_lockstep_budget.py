"""The lockstep Laplace solver's step budget.

A caller with a part of the SMs takes the lockstep launches from fewer
right-hand sides on, and these run a fixed number of refinement cycles.
Whatever restart length, tolerance and right-hand sides the caller has, a
solve that the persistent kernel finishes ends below the tolerance there too:
the bound is the tolerance itself.
"""
import numpy as np
import pytest

from mke_gb300 import phelm, serve

pytestmark = pytest.mark.gpu


def right_hand_sides(m, kind, nv):
    rng = np.random.default_rng(17)
    if kind == "points":      # one point each
        F = np.zeros((nv, m.size))
        F[np.arange(nv), rng.integers(0, m.size, nv)] = 1.0
        return F
    if kind == "constant":
        return np.outer(np.arange(1.0, nv + 1), np.ones(m.size))
    if kind == "noise":
        return rng.standard_normal((nv, m.size))
    return serve.solve_inputs(*m.latlon(), nv, seed=23)


@pytest.mark.parametrize("level,nv,sms,restart,tol,kind", [
    (3, 40, 2, 4, 1e-12, "smooth"), (4, 40, 8, 4, 1e-12, "smooth"), (4, 40, 8, 2, 1e-12, "smooth"),
    (5, 20, 8, 7, 1e-12, "smooth"), (4, 40, 8, 8, 1e-12, "constant"), (4, 40, 8, 30, 1e-12, "constant"),
    (5, 40, 40, 30, 1e-13, "points"), (6, 16, 16, 30, 1e-12, "points"), (7, 16, 40, 30, 1e-12, "noise")])
def test_capped_solves_reach_the_tolerance(level, nv, sms, restart, tol, kind):
    m = phelm.Mesh.sphere(level)
    F = right_hand_sides(m, kind, nv)
    ops = phelm.Operators(m, phelm.PHG_MIXED, restart=restart, tol=tol)
    ops.set_sms(sms)
    phelm.SphereLaplace(ops).solve_batch(F)
    assert ops.last_solve()["relres"] <= tol
