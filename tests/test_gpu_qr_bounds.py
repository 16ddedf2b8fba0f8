"""The per-sector QR is orthogonal and exact to a few N eps (Frobenius): Q is a product of N reflectors, which
round by eps each in directions of their own.  Sectors with fewer rows than a warp has lanes, and with row
counts that leave its lanes unequal work."""
import numpy as np
import pytest

from tests.test_gpu_qr_cluster import EPS, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shapes", [[(2, 1), (5, 3), (9, 9), (33, 7), (130, 8)], [(129, 17), (300, 82), (67, 66)],
                                    [(257, 129)], [(1000, 90)], [(240, 230)]])
@pytest.mark.parametrize("direction", ["l", "r"])
def test_close(cuda_ctx, shapes, direction):
    for A, Q, R in run(cuda_ctx, shapes, direction, lambda rng, M, N: rng.standard_normal((M, N))):
        N = A.shape[1]
        tol = 4 * max(N, 2) * EPS
        assert np.linalg.norm(Q.T @ Q - np.eye(N)) <= tol
        assert np.linalg.norm(A - Q @ R) <= tol * np.linalg.norm(A)
        assert (np.tril(R, -1) == 0).all() and (np.diag(R) >= 0).all()
