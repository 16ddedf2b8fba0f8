"""The per-sector SVD's right singular vectors are orthogonal to N eps a pair, which is what its sweeps promise,
also where the last rotation met a pair that was only just not orthogonal enough.  Bound: N eps a pair, and
four roundings of the rotated and normalised columns."""
import numpy as np
import pytest

from tests.test_gpu_svd_cluster import EPS, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [2, 3, 5, 8])
def test_nearly_orthogonal_pairs(cuda_ctx, N):
    """Columns of R^T with |<b_i, b_j>| about 1e-8 |b_i| |b_j|: one rotation each is within its FP32 tangent's
    error of enough."""
    def make(rng, M, n):
        d = np.sort(rng.uniform(0.02, 1.0, n))[::-1]
        A = np.diag(d) + np.triu(rng.uniform(0.8e-8, 1.4e-8, (n, n)), 1) * np.sqrt(d[:, None] * d[None, :])
        return np.concatenate([A, np.zeros((M - n, n))])
    for A, U, S, V in run(cuda_ctx, [(2 * N, N)] * 400, "l", make):
        off = np.abs(V.T @ V - np.eye(N))
        assert off.max() <= (N + 4) * EPS, off.max() / EPS


def close(A, U, S, V):
    """Orthogonality and residual to a few N eps (Frobenius): U and V are products of N reflectors and some
    8 N rotations a column, which round by eps each in directions of their own; V's pairs by 16 eps besides."""
    N = A.shape[1]
    one, tol = np.eye(N), 4 * N * EPS
    assert np.linalg.norm(U.T @ U - one) <= tol
    assert np.linalg.norm(V.T @ V - one) <= tol + N * min(N, 16) * EPS
    assert np.linalg.norm(A - (U * S) @ V.T) <= tol * np.linalg.norm(A)
    assert np.abs(S - np.linalg.svd(A, compute_uv=False)).max() <= tol * S[0]


# to the widest square sector that a cluster holds, and the first that it does not
@pytest.mark.parametrize("shapes", [[(9, 8), (31, 15), (17, 17), (40, 33)], [(136, 68), (331, 82)], [(200, 97), (118, 118)],
                                    [(300, 200)], [(244, 244)]])
@pytest.mark.parametrize("decades", [0, 6])
def test_close(cuda_ctx, shapes, decades):
    def make(rng, M, N):
        return (rng.standard_normal((M, N)) * np.logspace(0, -decades, N)) @ rng.permutation(np.eye(N))
    for out in run(cuda_ctx, shapes, "l", make):
        close(*out)


def test_first_sector_past_the_cluster(cuda_ctx):
    """The global-memory form: pairs of U's columns to M eps, V a product of rotations."""
    for A, U, S, V in run(cuda_ctx, [(245, 245)], "r", lambda rng, M, N: rng.standard_normal((M, N))):
        one, tol = np.eye(245), 245 * 245 * EPS
        assert np.linalg.norm(U.T @ U - one) <= tol and np.linalg.norm(V.T @ V - one) <= tol
        assert np.linalg.norm(A - (U * S) @ V.T) <= tol * np.linalg.norm(A)
