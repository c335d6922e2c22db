"""The level-by-level multigrid solver (gmres_kernel).

It runs where a V-cycle has more than one sweep a side (PHG_MG_NU=2 at
operator creation): one Laplacian, the baroclinic block system and, with
PHG_MG_CLUSTER=8, the coarse levels inside a thread-block cluster.  The
kernel's phase line (PHG_PHASE_TIMING) names the cluster it was launched with,
so each test sees that the path it is about ran.  Two solvers' results at
1e-12 agree to 1e-9, as everywhere; with and without the cluster the
arithmetic is the same, so the bits are.
"""
import numpy as np
import pytest

from mke_gb300 import fields, phelm, serve

pytestmark = pytest.mark.gpu

PRECISIONS = pytest.mark.parametrize("precision", [phelm.PHG_FP64, phelm.PHG_MIXED], ids=["fp64", "mixed"])


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def two_sweeps(m, precision, monkeypatch, cluster=0):
    with monkeypatch.context() as mp:
        mp.setenv("PHG_MG_NU", "2")
        mp.setenv("PHG_MG_CLUSTER", str(cluster))
        return phelm.Operators(m, precision, tol=1e-12)


def phase_lines(capfd, n):
    return [line for line in capfd.readouterr().err.splitlines() if line.startswith(f"[phases] n={n} ")]


@PRECISIONS
def test_cluster_tail_ran_and_equals_group_levels(precision, monkeypatch, capfd):
    m = phelm.Mesh.sphere(6)
    F = serve.solve_inputs(*m.latlon(), 1, seed=21)[0]
    monkeypatch.setenv("PHG_ROWS_PER_BLOCK", "257")   # 160 blocks, whole clusters, either way
    monkeypatch.setenv("PHG_PHASE_TIMING", "1")
    got = []
    for cluster in (8, 0):
        ops = two_sweeps(m, precision, monkeypatch, cluster)
        capfd.readouterr()
        got.append(phelm.SphereLaplace(ops).solve(F))
        lines = phase_lines(capfd, m.inner_size)
        assert lines and all(f" cluster={cluster} " in line for line in lines), lines
        assert ops.last_solve()["relres"] <= 1e-12
    assert np.array_equal(got[0].view(np.uint64), got[1].view(np.uint64))


@PRECISIONS
@pytest.mark.parametrize("level,nv", [(3, 1), (4, 9), (5, 3)])
def test_laplacian_matches_the_default_solver(level, nv, precision, monkeypatch, capfd):
    m = phelm.Mesh.sphere(level)
    F = serve.solve_inputs(*m.latlon(), nv, seed=22)
    want = phelm.SphereLaplace(phelm.Operators(m, precision, tol=1e-12)).solve_batch(F)
    ops = two_sweeps(m, precision, monkeypatch)
    monkeypatch.setenv("PHG_PHASE_TIMING", "1")
    capfd.readouterr()
    got = phelm.SphereLaplace(ops).solve_batch(F)
    assert phase_lines(capfd, m.inner_size)
    assert ops.last_solve()["relres"] <= 1e-12
    assert all(rel(a, b) <= 1e-9 for a, b in zip(got, want))


@PRECISIONS
def test_block_system_matches_the_default_solver(precision, monkeypatch, capfd):
    m = phelm.Mesh.sphere(4)
    lat, lon = m.latlon()
    u = [fields.barvortex_initial(lat, lon, seed=k)[0] for k in (31, 32)]
    want = phelm.Baroclin(phelm.Operators(m, precision, tol=1e-12), coriolis=np.sin(lat)).calc(*u)
    bc = phelm.Baroclin(two_sweeps(m, precision, monkeypatch), coriolis=np.sin(lat))
    monkeypatch.setenv("PHG_PHASE_TIMING", "1")
    capfd.readouterr()
    got = bc.calc(*u)
    assert phase_lines(capfd, 4 * m.inner_size)
    assert all(rel(a, b) <= 1e-9 for a, b in zip(got, want))
