"""The adjoint step at levels 6 and 7 against values recorded on a GB300.

BarVortex::calc_LT (examples/barvortex_impl.h:485-535) solves with the step's
matrix and then applies the Laplacian.  What the solve's stopping test leaves
of the residual (1e-12, grid-scale in mixed precision) is amplified by the
ratio of the largest eigenvalue of M^-1 L to the field's: about 5e4 / 60 at
level 6, so the mixed result is determined to 1e-9 there and to 4 times that
at level 7.  tests/golden/adjoint_gpu.npz holds every 37th value of the
results that this library gave with its group-barrier solvers; the bound is
the one every solve-based result keeps, 1e-9 relative.
"""
import numpy as np
import pytest

from mke_gb300 import fields, phelm

pytestmark = pytest.mark.gpu

STRIDE = 37


def adjoint(level, precision):
    m = phelm.Mesh.sphere(level)
    lat, lon = m.latlon()
    bv = phelm.BarVortex(phelm.Operators(m, precision, tol=1e-12), tau=1e-3, sigma=1.6e-2, mu=8e-5, theta=0.5,
                         picard_iters=3, coriolis=np.sin(lat))
    c = fields.random_coeffs(np.random.default_rng(13), 1, 12, 0.05)
    v = fields.sh_field(fields.sh_inverse_laplacian(c), lat, lon)
    z, _ = fields.barvortex_initial(lat, lon, seed=14, lmax_noise=16)
    return bv.calc_LT(v, z)


@pytest.mark.parametrize("precision", [phelm.PHG_FP64, phelm.PHG_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("level", [6, 7])
def test_adjoint_as_recorded(golden, level, precision):
    want = golden("adjoint_gpu.npz")[f"L{level}_{'mixed' if precision == phelm.PHG_MIXED else 'fp64'}"]
    got = adjoint(level, precision)[::STRIDE]
    assert np.linalg.norm(got - want) <= 1e-9 * np.linalg.norm(want)
