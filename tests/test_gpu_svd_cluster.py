"""The per-sector SVD at the sizes where its work split changes: fewer columns than CTAs of a cluster or
column blocks, one more or less than a multiple, products in one piece or several, U in shared or global
memory, sectors too large for a cluster; graded and rank-deficient sectors.  Bounds (Frobenius norm):
U is a product of reflectors and rotations, |U^T U - 1| and |A - U S V^T| / |A| stay within a few
N sqrt(M N) eps, singular values differ from LAPACK's by no more; the columns of V are orthogonal to the
sweeps' N eps a pair, N^2 eps in all, and to their own rounding."""
import numpy as np
import pytest

from imps_cpp_tools_gb300 import blocks as B
from imps_cpp_tools_gb300 import ops

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52


def dev(a):
    import torch
    return torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def run(ctx, shapes, direction, make):
    """shapes: (M, N) per sector, two blocks of rows each; returns (A, U, S, V) per sector, tall form."""
    rng = np.random.default_rng(sum(m * 31 + n for m, n in shapes))
    blocks, parts, mats = [], [], [make(rng, M, N) for M, N in shapes]
    for s in (0, 1):
        for q, (M, N) in enumerate(shapes):
            rows = mats[q][:M // 2] if s == 0 else mats[q][M // 2:]
            other = 1000 * (s + 1) + q
            if direction == "l":
                blocks.append((s, (other,), (q,), rows.shape[0], N))
                parts.append(rows)
            else:
                blocks.append((s, (q,), (other,), N, rows.shape[0]))
                parts.append(rows.T)
    lay = B.Layout(blocks, 1)
    dec = B.plan_decomp(ctx, lay, direction)
    flat = np.concatenate([p.reshape(-1, order="F") for p in parts])
    n = sum(N for _, N in shapes)
    U, S, V = (dev(np.full(k, np.nan)) for k in (lay.nelem, n, dec.rlayout.nelem))
    assert ops.svd(dec, dev(flat), U, S, V)
    Uh, Sh, Vh = (x.cpu().numpy() for x in (U, S, V))
    out, o, so = [], 0, 0
    for q, (M, N) in enumerate(shapes):
        v = Vh[o:o + N * N].reshape(N, N, order="F")
        s = Sh[so:so + N]
        o, so = o + N * N, so + N
        halves = []
        for k in (0, 1):
            i = k * len(shapes) + q
            (_, _, _, rows, cols), off = lay.blocks[i], lay.offsets[i]
            h = Uh[off:off + rows * cols].reshape(rows, cols, order="F")
            halves.append(h if direction == "l" else h.T)
        out.append((mats[q], np.concatenate(halves), s, v.T if direction == "l" else v))
    return out


def check(A, U, S, V, full_rank=True):
    M, N = A.shape
    tol = 4 * np.sqrt(M * N) * N * EPS
    one = np.eye(N)
    assert np.isfinite(U).all() and np.isfinite(S).all() and np.isfinite(V).all()
    assert (np.diff(S) <= 0).all() and (S >= 0).all()
    assert np.linalg.norm(U.T @ U - one) <= tol
    if full_rank:
        assert np.linalg.norm(V.T @ V - one) <= tol + N * N * EPS
    norm = max(np.linalg.norm(A), 1e-300)
    assert np.linalg.norm(A - (U * S) @ V.T) <= tol * norm
    assert np.abs(S - np.linalg.svd(A, compute_uv=False)).max() <= tol * norm


SHAPES = [[(1, 1)], [(3, 2), (7, 7), (8, 8), (9, 8), (17, 9), (16, 16), (31, 15), (17, 17)],
          [(40, 33), (331, 82), (136, 68), (65, 64)], [(96, 96), (200, 97)], [(118, 118), (272, 136)], [(700, 100)],
          [(450, 200), (5, 3)], [(230, 230)], [(3000, 90)], [(2000, 110)],
          [(300, 257)], [(4 + i % 3, 1 + i % 4) for i in range(300)]]


@pytest.mark.parametrize("shapes", SHAPES)
@pytest.mark.parametrize("direction", ["l", "r"])
def test_shapes(cuda_ctx, shapes, direction):
    for A, U, S, V in run(cuda_ctx, shapes, direction, lambda rng, M, N: rng.standard_normal((M, N))):
        check(A, U, S, V)


@pytest.mark.parametrize("scale", [1.0, 1e-100, 1e100])
@pytest.mark.parametrize("decades", [12, 40])
def test_graded(cuda_ctx, scale, decades):
    """Singular values over many decades, as a centre matrix's sectors near convergence."""
    def make(rng, M, N):
        return scale * (rng.standard_normal((M, N)) * np.logspace(0, -decades, N)) @ rng.permutation(np.eye(N))
    for A, U, S, V in run(cuda_ctx, [(136, 68), (20, 9)], "l", make):
        check(A / scale, U, S / scale, V)


def test_rank_deficient(cuda_ctx):
    def make(rng, M, N):
        k = N // 3
        return rng.standard_normal((M, k)) @ rng.standard_normal((k, N))
    for A, U, S, V in run(cuda_ctx, [(136, 68), (20, 9), (6, 6)], "l", make):
        check(A, U, S, V, full_rank=False)
    for A, U, S, V in run(cuda_ctx, [(30, 20), (1, 1)], "r", lambda rng, M, N: np.zeros((M, N))):
        check(A, U, S, V, full_rank=False)
    for A, U, S, V in run(cuda_ctx, [(30, 20)], "r", lambda rng, M, N: np.eye(M, N)):
        check(A, U, S, V)
