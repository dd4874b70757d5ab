"""The LU and the solves at their edges (the shared-memory kernel up to 116 rows;
16-column register panels, 128-column blocks, one to several CTAs per panel;
32-row quarters of the triangles), through the star product's inverse, on matrices
whose pivots leave the diagonal."""
import numpy as np
import pytest

import openrcwa_b200 as o
from oracle.smatrix_oracle import star_product

pytestmark = pytest.mark.gpu


def _inverses(eng, A):
    """(I - A)^-1 of every item, through the star product's Tdd with unit Tdd, Rud and tdd."""
    I, Z = np.broadcast_to(np.eye(A.shape[-1], dtype=complex), A.shape), np.zeros_like(A)
    got, st = eng.star_product({"Rud": I, "Rdu": Z, "Tdd": I, "Tuu": Z}, {"rud": Z, "rdu": A, "tdd": I, "tuu": Z})
    assert not np.any(st)
    return got["Tdd"]


# one, two and three CTAs per first panel as the rows need them
@pytest.mark.parametrize("n", [200, 529, 1058])
def test_panel_clusters_give_identical_factors(n):
    rng = np.random.default_rng(n)
    A = (rng.standard_normal((2, n, n)) + 1j * rng.standard_normal((2, n, n))) / np.sqrt(n)
    eng = o.Engine(0)
    try:
        o.set_lu_cluster(0)
        X = _inverses(eng, A)
        for team in (4, 8):
            o.set_lu_cluster(team)
            assert o.lu_cluster_size(n, 2) == team
            assert np.array_equal(_inverses(eng, A), X), team
    finally:
        o.set_lu_cluster(0)
        eng.close()
    res = np.linalg.norm((np.eye(n) - A) @ X - np.eye(n)) / np.linalg.norm(X)
    # residual of an inverse from an LU: a modest multiple of n u |A| |X|
    assert res <= 40 * n * 2.0 ** -53 * np.linalg.norm(np.eye(n) - A)


def test_panels_above_the_register_rows():
    # above 4096 rows: 32-column panels updated in L2, by one CTA and by a team
    n = 4101
    rng = np.random.default_rng(7)
    A = (rng.standard_normal((1, n, n)) + 1j * rng.standard_normal((1, n, n))) / np.sqrt(n)
    eng = o.Engine(0)
    try:
        o.set_lu_cluster(1)
        X = _inverses(eng, A)
        o.set_lu_cluster(0)
        assert o.lu_cluster_size(n, 1) > 1
        assert np.array_equal(_inverses(eng, A), X)
    finally:
        o.set_lu_cluster(0)
        eng.close()
    v = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    x = X[0] @ v
    # residual bound of a solve: a modest multiple of n u |A| |x|
    norm_a = np.linalg.norm(np.eye(n) - A[0])
    assert np.linalg.norm(x - A[0] @ x - v) <= 40 * n * 2.0 ** -53 * norm_a * np.linalg.norm(x)


@pytest.mark.parametrize("n,batch", [(1, 2), (2, 1), (15, 2), (16, 2), (17, 3), (31, 2), (33, 2), (64, 1),
                                     (98, 3), (115, 2), (116, 2), (117, 2), (129, 2), (143, 3), (144, 1), (145, 2), (255, 1), (257, 2), (400, 2), (513, 1),
                                     (529, 2), (1030, 1),
                                     # more 64-column slabs than SMs: blocked solves at every order
                                     (16, 149), (17, 149), (33, 149), (66, 75), (98, 75), (117, 75)])
def test_star_product_inverse(n, batch):
    rng = np.random.default_rng(n)

    def rand(scale=1.0):
        return scale * (rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n)))

    S = {k: rand(1.0 / np.sqrt(n)) for k in ("Rud", "Rdu", "Tdd", "Tuu")}
    s = {k: rand(1.0 / np.sqrt(n)) for k in ("rud", "rdu", "tdd", "tuu")}
    eng = o.Engine(0)
    got, st = eng.star_product(S, s)
    eng.close()
    assert not np.any(st)
    for b in range(batch):
        Sb, sb = {k: v[b] for k, v in S.items()}, {k: v[b] for k, v in s.items()}
        ref = star_product(Sb, sb)
        # forward error of the inverse: its condition number times n u
        cond = np.linalg.cond(np.eye(n) - sb["rdu"] @ Sb["Rud"])
        for k in ref:
            err = np.linalg.norm(got[k][b] - ref[k]) / np.linalg.norm(ref[k])
            assert err <= 4 * n * 2.0 ** -53 * cond, (k, err, cond)
