"""phg_ops_validate reads the time steppers' index tables too: more checks run
once a handle has steppers (their forward and, from the first inverse
linearised step on, backward systems), none of them finds an entry out of
range, and a destroyed stepper's tables are left alone."""
import numpy as np
import pytest

from mke_gb300 import phelm, serve

pytestmark = pytest.mark.gpu


def checks(ops):
    k0 = phelm.kernel_launches()
    assert ops.validate() == 0
    return phelm.kernel_launches() - k0


@pytest.mark.parametrize("precision", [phelm.PHG_FP64, phelm.PHG_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("level", [2, 3, 5])
def test_steppers_tables_are_checked(level, precision):
    m = phelm.Mesh.sphere(level)
    lat, lon = m.latlon()
    u = serve.solve_inputs(lat, lon, 4, seed=9)
    ops = phelm.Operators(m, precision, tol=1e-12)
    alone = checks(ops)
    bv = phelm.BarVortex(ops, coriolis=np.sin(lat))
    forward = checks(ops)
    assert forward > alone                      # D^-1 A of the step's matrix
    bv.calc_L_1(u[0], u[1])
    assert checks(ops) > forward                # and of the backward one
    bc = phelm.Baroclin(ops, coriolis=np.sin(lat))
    both = checks(ops)
    bc.calc_L_1(u[0], u[1], u[2], u[3])
    # the block system's columns, and with a hierarchy (level 3 on) its composed table
    assert checks(ops) - both == (2 if level >= 3 else 1)
    del bv, bc
    assert checks(ops) == alone
