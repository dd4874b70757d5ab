"""The LU and the solves at their edges (the shared-memory kernel up to 116 rows;
16-column register panels, 128-column blocks, one to several CTAs per panel;
32-row quarters of the triangles), through the star product's inverse, on matrices
whose pivots leave the diagonal."""
import numpy as np
import pytest

import openrcwa_b200 as o
from oracle.smatrix_oracle import star_product

pytestmark = pytest.mark.gpu


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
