"""The persistent multigrid solver of the Laplacian (phg_mgs.cu) at the shapes
where its row split, its shared-memory plan and its dense coarse product
change: the smallest mesh with a hierarchy (dense from the finest level), the
next ones (dense from one and two levels down), one block, a few and all SMs
per right-hand side, more right-hand sides than SMs, and short restarts.

Reference: scipy's sparse LU of the same assembled matrix.  Both solutions are
the discrete one up to (condition number) x (relative residual): 1e-12 times
about 1e3 at these levels, and the LU's 1e-16 times that; 1e-9 is the bound of
every solve-based comparison here.
"""
import functools

import numpy as np
import pytest

from mke_gb300 import phelm, serve

pytestmark = pytest.mark.gpu


@functools.lru_cache(maxsize=None)
def problem(level, count):
    sp = pytest.importorskip("scipy.sparse")
    from scipy.sparse.linalg import splu
    m = phelm.Mesh.sphere(level)
    lat, lon = m.latlon()
    F = serve.solve_inputs(lat, lon, count, seed=77)
    bnd = np.random.default_rng(5).standard_normal((count, m.outer_size))

    def mat(name, cols):
        ptr, col, val = m.csr(name)
        return sp.csr_matrix((val, col, ptr), shape=(m.inner_size, cols))

    inner = m.maps()["inner"]
    b = mat("idt", m.inner_size) @ F[:, inner].T + mat("bnd2", m.outer_size) @ bnd.T
    x = splu(mat("lapl", m.inner_size).tocsc()).solve(b)
    return m, F, bnd, inner, x.T


def check(m, ops, F, bnd, inner, want):
    got = phelm.SphereLaplace(ops).solve_batch(F, bnd)
    assert ops.last_solve()["relres"] <= 1e-12
    for k in range(len(F)):
        assert np.linalg.norm(got[k][inner] - want[k]) <= 1e-9 * np.linalg.norm(want[k]), k
        assert np.array_equal(np.delete(got[k], inner), bnd[k])


@pytest.mark.parametrize("precision", [phelm.PHG_FP64, phelm.PHG_MIXED])
@pytest.mark.parametrize("level", [3, 4, 5])
@pytest.mark.parametrize("sms", [0, 1, 2, 40])
def test_blocks_per_right_hand_side(level, precision, sms):
    m, F, bnd, inner, want = problem(level, 3)
    ops = phelm.Operators(m, precision, tol=1e-12)
    ops.set_sms(sms)
    check(m, ops, F, bnd, inner, want)
    check(m, ops, F[:1], bnd[:1], inner, want)


@pytest.mark.parametrize("precision", [phelm.PHG_FP64, phelm.PHG_MIXED])
def test_more_right_hand_sides_than_sms(precision):
    m, F, bnd, inner, want = problem(3, 320)
    check(m, phelm.Operators(m, precision, tol=1e-12), F, bnd, inner, want)


@pytest.mark.parametrize("precision", [phelm.PHG_FP64, phelm.PHG_MIXED])
@pytest.mark.parametrize("restart", [1, 7, 8, 9, 48])
def test_restarts(precision, restart):
    m, F, bnd, inner, want = problem(4, 1)
    ops = phelm.Operators(m, precision, restart=restart, tol=1e-12)
    check(m, ops, F, bnd, inner, want)


def test_rows_per_block(monkeypatch):
    m, F, bnd, inner, want = problem(5, 1)
    ops = phelm.Operators(m, phelm.PHG_MIXED, tol=1e-12)
    for rows in ("64", "1000", "20000"):
        monkeypatch.setenv("PHG_ROWS_PER_BLOCK", rows)
        check(m, ops, F, bnd, inner, want)


@pytest.mark.parametrize("precision", [phelm.PHG_FP64, phelm.PHG_MIXED])
@pytest.mark.parametrize("level", [2, 3, 4, 5])
@pytest.mark.parametrize("members,sms", [(1, 0), (2, 1), (3, 0), (3, 7), (5, 150), (9, 0), (160, 0)])
def test_mass_solves(level, precision, members, sms):
    """The persistent Chebyshev solver (phg_chs.cu) through the barotropic
    step: members (so 1 to 1,280 right-hand sides a solve, chunks of 1, 2, 4
    and 8) over one, a few and all SMs, against the members' own single steps;
    both solve to 1e-12, and 1e-9 is the bound of every step comparison."""
    if members == 160 and level > 3:
        pytest.skip("covered by the smaller meshes")
    m = phelm.Mesh.sphere(level)
    lat, lon = m.latlon()
    u = serve.barvortex_inputs(lat, lon, members, seed=9)
    ops = phelm.Operators(m, precision, tol=1e-12)
    bv = phelm.BarVortex(ops, coriolis=np.sin(lat))
    single = {k: bv.calc(u[k]) for k in {0, members // 2, members - 1}}
    ops.set_sms(sms)
    got = bv.calc_batch(u)
    for k, want in single.items():
        assert np.linalg.norm(got[k] - want) <= 1e-9 * np.linalg.norm(want), k
