"""The per-sector QR at the sizes where its work split changes: fewer columns than CTAs of a cluster, one
more or less than a multiple, Q in shared or global memory, sectors too large for a cluster's shared
memory; and rank-deficient sectors.  Bounds: Householder QR is backward stable, |Q^T Q - 1| and
|A - Q R| / |A| stay within a few M N eps in the Frobenius norm; a full-rank, well-conditioned sector's
factors agree with LAPACK's to that times its condition number."""
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
    """shapes: (M, N) per sector, two blocks of rows each; returns (A, Q, R) per sector, tall form."""
    rng = np.random.default_rng(sum(m * 31 + n for m, n in shapes))
    blocks, parts, mats = [], [], []
    # direction l: blocks (s, qin -> qout = sector) stacked by rows; r: (s, sector -> qout) by columns
    for s in (0, 1):
        for q, (M, N) in enumerate(shapes):
            if s == 0:
                mats.append(make(rng, M, N))
            cut = M // 2
            rows = mats[q][:cut] if s == 0 else mats[q][cut:]
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
    Q, R = dev(np.full(lay.nelem, np.nan)), dev(np.full(dec.rlayout.nelem, np.nan))
    ops.qr(dec, dev(flat), Q, R)
    ctx.synchronize()
    Qh, Rh = Q.cpu().numpy(), R.cpu().numpy()
    out, o = [], 0
    for q, (M, N) in enumerate(shapes):
        r = Rh[o:o + N * N].reshape(N, N, order="F")
        o += N * N
        halves = []
        for s in (0, 1):
            i = s * len(shapes) + q
            (_, _, _, rows, cols), off = lay.blocks[i], lay.offsets[i]
            h = Qh[off:off + rows * cols].reshape(rows, cols, order="F")
            halves.append(h if direction == "l" else h.T)
        out.append((mats[q], np.concatenate(halves), r if direction == "l" else r.T))
    return out


def check(A, Q, R, unique):
    M, N = A.shape
    tol = 4 * np.sqrt(M * N) * N * EPS
    assert np.isfinite(Q).all() and np.isfinite(R).all()
    assert np.linalg.norm(Q.T @ Q - np.eye(N)) <= tol
    assert np.linalg.norm(A - Q @ R) <= tol * max(np.linalg.norm(A), 1e-300)
    assert (np.tril(R, -1) == 0).all() and (np.diag(R) >= 0).all()
    if unique:
        q, r = np.linalg.qr(A)
        sg = np.where(np.diag(r) < 0, -1.0, 1.0)
        cond = np.linalg.cond(A)
        assert np.linalg.norm(Q - q * sg) <= 4 * cond * tol
        assert np.linalg.norm(R - r * sg[:, None]) <= 4 * cond * tol * np.linalg.norm(A)


SHAPES = [[(1, 1)], [(3, 2), (7, 7), (8, 8), (9, 8), (17, 9), (16, 16)], [(40, 33), (331, 82), (136, 68), (65, 64)],
          [(700, 150)], [(2000, 96)], [(404, 404)], [(600, 512), (20, 5)]]


@pytest.mark.parametrize("shapes", SHAPES)
@pytest.mark.parametrize("direction", ["l", "r"])
def test_shapes(cuda_ctx, shapes, direction):
    for A, Q, R in run(cuda_ctx, shapes, direction, lambda rng, M, N: rng.standard_normal((M, N))):
        check(A, Q, R, True)


@pytest.mark.parametrize("direction", ["l", "r"])
def test_graded(cuda_ctx, direction):
    """Columns over twelve decades, as a centre matrix's sectors near convergence."""
    make = lambda rng, M, N: rng.standard_normal((M, N)) * np.logspace(0, -12, N)
    for A, Q, R in run(cuda_ctx, [(136, 68), (20, 9)], direction, make):
        check(A, Q, R, False)
        # column by column: |a_j - Q r_j| relative to that column
        err = np.linalg.norm(A - Q @ R, axis=0) / np.linalg.norm(A, axis=0)
        assert (err <= 4 * np.sqrt(A.size) * EPS * A.shape[1]).all()


@pytest.mark.parametrize("kind", ["zero", "zero column", "equal columns", "first rows only"])
def test_rank_deficient(cuda_ctx, kind):
    def make(rng, M, N):
        A = rng.standard_normal((M, N))
        if kind == "zero":
            A[:] = 0.0
        elif kind == "zero column":
            A[:, N // 2] = 0.0
        elif kind == "equal columns":
            A[:, -1] = A[:, 0]
        else:
            A = np.triu(A)
        return A
    for A, Q, R in run(cuda_ctx, [(30, 12), (9, 9), (100, 41)], "l", make):
        check(A, Q, R, False)
