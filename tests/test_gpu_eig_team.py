"""The eigensolver with a team (thread-block cluster) of CTAs per matrix
(rcwa_set_eig_cluster): the team splits the rows of the Hessenberg panel
products, the tiles of its GEMMs and the off-window lines of the Schur sweeps,
and every element is computed by the same operations as with one CTA, so the
eigenvalues and eigenvectors are identical bit for bit for every team size."""
import numpy as np
import pytest

import openrcwa_b200 as o

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    e = o.Engine(0)
    yield e
    o.set_eig_cluster(0)
    e.close()


def _matrices(n, b, seed):
    rng = np.random.default_rng(seed)
    return rng.normal(size=(b, n, n)) + 1j * rng.normal(size=(b, n, n))


@pytest.mark.parametrize("n,b", [(200, 3), (450, 2)])
def test_team_sizes_give_identical_results(eng, n, b):
    A = _matrices(n, b, n)
    o.set_eig_cluster(1)
    w1, V1, i1 = eng.zgeev(A)
    assert not np.any(i1)
    for team in (2, 3, 8):
        o.set_eig_cluster(team)
        assert o.eig_cluster_size(n, b) == team
        w, V, info = eng.zgeev(A)
        assert not np.any(info)
        assert np.array_equal(w, w1) and np.array_equal(V, V1), team
    o.set_eig_cluster(0)
    for k in range(b):
        res = np.abs(A[k] @ V1[k] - V1[k] * w1[k][None, :]).max() / np.abs(A[k]).max()
        assert res < 1e-11


@pytest.mark.parametrize("log2max", [100.9, 101.1, -99.9, -100.1])
def test_teams_agree_beside_the_scaling_bounds(eng, log2max):
    # the reduction scales a matrix whose largest component has an exponent
    # outside [-100, 100]; at 100.9 it does not, but the first reflector's beta
    # (the norm of a column) lies above the bound, so a CTA that still scanned
    # after the first one had written beta would decide otherwise
    n = 200
    A = _matrices(n, 2, 11)
    A *= 2.0 ** log2max / max(np.abs(A.real).max(), np.abs(A.imag).max())
    o.set_eig_cluster(1)
    w1, V1, i1 = eng.zgeev(A)
    for team in (2, 8):
        o.set_eig_cluster(team)
        w, V, info = eng.zgeev(A)
        assert np.array_equal(info, i1) and np.array_equal(w, w1) and np.array_equal(V, V1), team
    o.set_eig_cluster(0)
    assert not np.any(i1)
    # backward error of a QR iteration: a modest multiple of n u |A|
    for k in range(2):
        assert np.linalg.norm(A[k] @ V1[k] - V1[k] * w1[k]) <= 40 * n * 2.0 ** -53 * np.linalg.norm(A[k])


def test_automatic_team_for_few_large_matrices(eng):
    o.set_eig_cluster(0)
    assert 2 <= o.eig_cluster_size(882, 4) <= 8
    assert o.eig_cluster_size(200, 4) == 3        # a CTA per 64 rows
    assert o.eig_cluster_size(1200, 148) == 1     # the batch fills the GPU
    assert o.eig_cluster_size(116, 4) == 1        # held in shared memory
    team = o.eig_cluster_size(1200, 4)
    assert 2 <= team <= 8
    A = _matrices(1200, 4, 7)
    w, V, _ = eng.zgeev(A)
    o.set_eig_cluster(1)
    w1, V1, _ = eng.zgeev(A)
    o.set_eig_cluster(0)
    assert np.array_equal(w, w1) and np.array_equal(V, V1)


def test_reported_sizes_are_those_of_the_launches(eng):
    # orders in shared memory take one CTA whatever is forced
    o.set_eig_cluster(8)
    try:
        assert [o.eig_cluster_size(n, 4) for n in (14, 64, 116, 117)] == [1, 1, 1, 8]
    finally:
        o.set_eig_cluster(0)
    # LU: one CTA for the whole matrix, then a CTA per 512 rows of the first
    # panel, or the forced size if that is larger
    o.set_lu_cluster(0)
    assert [o.lu_cluster_size(n, 2) for n in (98, 128, 200, 512, 513, 1058, 4096)] == [1, 1, 1, 1, 2, 3, 8]
    assert o.lu_cluster_size(882, 1200) == 1
    o.set_lu_cluster(2)
    try:
        assert [o.lu_cluster_size(n, 2) for n in (98, 200, 1058, 4097)] == [1, 2, 3, 2]
    finally:
        o.set_lu_cluster(0)


def test_team_size_asked_before_the_first_solve():
    # the query must not depend on (or, being kept, spoil) what a solve sets up
    import subprocess
    import sys
    code = ("import openrcwa_b200 as o; a = o.eig_cluster_size(882, 4); e = o.Engine(0); "
            "import numpy as np; e.zgeev(np.eye(130)[None] + 0j); print(a, o.eig_cluster_size(882, 4))")
    out = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    a, b = (int(x) for x in out.stdout.split())
    assert a == b and a >= 2


def test_solve_with_teams_matches_single_cta(eng):
    # one point of a 2D pillar grating at Nx = Ny = 11 (n = 1058): three layer
    # eigensolves with automatic teams and LU panels on the three CTAs they
    # need, against one CTA per eigensolve and panels forced to eight; R, T and
    # every order must agree bit for bit
    from openrcwa_b200 import workloads
    stacks, pts, pxy = workloads.pillars_2d(seed=3, nH=11, n_lambda=1, n_angle=1, n_layers=3)
    o.set_eig_cluster(0)
    o.set_lu_cluster(0)
    assert o.eig_cluster_size(1058, 3) > 1 and o.lu_cluster_size(1058, 1) == 3
    R, T, REF, TRN, st = eng.solve_batch(stacks, pts[:1], pxy[:1])
    o.set_eig_cluster(1)
    o.set_lu_cluster(8)
    try:
        assert o.lu_cluster_size(1058, 1) == 8
        R1, T1, REF1, TRN1, st1 = eng.solve_batch(stacks, pts[:1], pxy[:1])
    finally:
        o.set_eig_cluster(0)
        o.set_lu_cluster(0)
    assert not np.any(st) and not np.any(st1)
    assert np.array_equal(R, R1) and np.array_equal(T, T1)
    assert np.array_equal(REF[0], REF1[0]) and np.array_equal(TRN[0], TRN1[0])
    assert np.all(R + T <= 1.0 + 1e-9)  # lossy layers
