"""The pipelined FP64 tile product at the edges of its tiles, blocks and slabs."""
import numpy as np
import pytest

import openrcwa_b200 as o

pytestmark = pytest.mark.gpu

# one element; below, at and above a block (8), a warp's share (32), a tile
# (64); K below, at and above a slab (8), the pipeline's depth (4 slabs) and an
# odd remainder; more than one tile each way
SIZES = [(1, 1, 1), (7, 9, 3), (8, 8, 8), (33, 31, 9), (63, 65, 31), (64, 64, 32), (65, 129, 33), (130, 1, 200),
         (98, 98, 98)]


@pytest.mark.parametrize("M,N,K", SIZES)
def test_zgemm_edges(M, N, K):
    rng = np.random.default_rng(M * 1000 + N * 10 + K)

    def rand(*s):
        return rng.standard_normal(s) + 1j * rng.standard_normal(s)

    A, B, C = rand(3, M, K), rand(3, K, N), rand(3, M, N)
    alpha, beta = 0.7 - 0.4j, -1.3 + 0.2j
    eng = o.Engine(0)
    plain = eng.zgemm(A, B)
    full = eng.zgemm(A, B, C, alpha, beta)
    eng.close()
    # elementwise bound of a K-term complex dot product: 4 (K + 4) u sum |a||b|
    bound = 4 * (K + 4) * 2.0 ** -53 * (np.abs(A) @ np.abs(B))
    assert np.all(np.abs(plain - A @ B) <= 2 * bound)
    ref = alpha * (A @ B) + beta * C
    assert np.all(np.abs(full - ref) <= 2 * (np.abs(alpha) * bound + 8 * 2.0 ** -53 * np.abs(beta) * np.abs(C)) + 1e-300)
