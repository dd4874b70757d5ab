"""The Schur kernels at their size edges: the shared-memory kernel (up to 116
rows, in steps of 32 per lane), the windowed multishift kernel with its chase
window (72) and early-deflation window (12), and the automatic teams of CTAs."""
import numpy as np
import pytest

import openrcwa_b200 as o

pytestmark = pytest.mark.gpu


def _cases(n, rng):
    R = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    yield R
    yield R + R.conj().T
    yield np.roll(np.eye(n), 1, axis=0).astype(complex)          # unreduced, equal moduli
    yield R * np.logspace(0, -12, n)[:, None]                    # graded
    H = np.triu(R, -1)
    if n > 2:
        H[n // 2, n // 2 - 1] = 0.0                              # already reducible
    yield H
    yield np.zeros((n, n), dtype=complex)


def _scales(R):
    # a matrix whose largest component's exponent lies outside [-100, 100] is
    # reduced, iterated and back-substituted at a power of two of its size: just
    # inside and outside the bounds, and to the ends of the range, where products
    # of the entries leave it and (at 1e-300) the entries lie below LAPACK's
    # smallest divisor of the back substitution
    top = max(np.abs(R.real).max(), np.abs(R.imag).max())
    yield from (2.0 ** 100.9 / top, 2.0 ** 101.1 / top, 2.0 ** -99.9 / top, 2.0 ** -100.1 / top)
    yield from (1e120, 1e-120, 1e150, 1e-150, 1e300, 1e-300)


@pytest.mark.parametrize("n", [1, 2, 3, 4, 7, 8, 31, 32, 33, 63, 64, 65, 96, 97, 115, 116, 117, 129, 150])
def test_schur_edges(n):
    rng = np.random.default_rng(n)
    A = list(_cases(n, rng))
    R = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    scale = np.array([1.0] * len(A) + list(_scales(R)))
    A = np.array(A + [R] * (len(scale) - len(A)))
    eng = o.Engine(0)
    w, V, info = eng.zgeev(A * scale[:, None, None])
    eng.close()
    assert not np.any(info)
    for a, ww, v in zip(A, w / scale[:, None], V):
        # backward error of a QR iteration: a modest multiple of n u |A|
        assert np.linalg.norm(a @ v - v * ww) <= 40 * n * 2.0 ** -53 * max(np.linalg.norm(a), 1e-300)
        assert np.allclose(np.linalg.norm(v, axis=0), 1.0, atol=1e-12)
