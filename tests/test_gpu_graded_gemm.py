"""The FP64 grouped GEMM where its operands are graded along k, rows and columns oppositely: every output keeps
the error bound of FP64 multiply-adds, which is relative to sum_k |a_ik| |b_kj| and not to the largest entries.
Bound, derived: digits dropped and cut off are below K 2^-53 of that sum (an output for which they might not be
is computed by multiply-adds, (K + 1) 2^-53), and every addition of chunks, shares, halves and lanes rounds by
2^-53 of it: at most 16 and 4 per term.  And the digit sums at the bound of what FP32 accumulators hold."""
import numpy as np
import pytest

from tests.test_gpu_split_gemm import one_block, run_program, stored

pytestmark = pytest.mark.gpu
ORDERS = [(0, 0), (1, 0), (0, 1), (1, 1)]


def check(got, mats, alphas):
    ref = np.zeros(got.shape, np.longdouble)
    mag = np.zeros(got.shape, np.longdouble)
    for (A, Bm), al in zip(mats, alphas):
        ref += al * (A.astype(np.longdouble) @ Bm.astype(np.longdouble))
        mag += abs(al) * (np.abs(A).astype(np.longdouble) @ np.abs(Bm).astype(np.longdouble))
    bound = (sum(A.shape[1] for A, _ in mats) + 16 + 4 * len(mats)) * np.longdouble(2.0) ** -53 * mag
    err = np.abs(got - ref)
    assert (err <= bound).all(), float((err / np.maximum(bound, np.longdouble(1e-4000))).max())


def graded(rng, M, Nn, K, decades):
    """A falling and B rising by `decades` along k."""
    g = 10.0 ** (-decades * np.arange(K) / max(K - 1, 1))
    return rng.standard_normal((M, K)) * g, rng.standard_normal((K, Nn)) * g[::-1, None]


@pytest.mark.parametrize("M,Nn,K", [(1, 1, 2), (16, 8, 17), (33, 31, 40), (68, 68, 68), (20, 82, 81), (40, 9, 300)])
@pytest.mark.parametrize("decades", [0, 2, 4, 8, 12, 20, 40])
def test_graded_along_k(cuda_ctx, M, Nn, K, decades):
    rng = np.random.default_rng(decades * 1000 + K)
    mats = [graded(rng, M, Nn, K, decades), graded(rng, M, Nn, max(1, K // 2), decades / 2)]
    for t in ORDERS:
        check(one_block(cuda_ctx, M, Nn, mats, [1.0, -0.75], [t, t], pad=1)[:M], mats, [1.0, -0.75])


@pytest.mark.parametrize("kind", ["selection", "diagonal", "rows", "sparse", "scattered"])
def test_uneven_operands(cuda_ctx, kind):
    rng = np.random.default_rng(11)
    n = 50
    A, Bm = rng.standard_normal((n, n)), rng.standard_normal((n, n))
    if kind == "selection":    # an identity with a negligible second entry in every row
        A = np.eye(n) + 2.0 ** -90 * np.roll(np.eye(n), 1, 1)
        Bm = Bm * 2.0 ** rng.integers(-300, 100, (n, n))
    elif kind == "diagonal":   # as an environment near its fixed point: a large diagonal
        A = 1e5 * np.eye(n) + A * 10.0 ** -rng.integers(0, 12, (n, n))
        Bm = Bm * 10.0 ** -rng.integers(0, 9, (n, n))
    elif kind == "rows":       # some outputs tiny among ordinary ones
        A[:, :25] *= 2.0 ** -40
        Bm[25:, ::3] *= 2.0 ** -45
    elif kind == "sparse":     # sums that are exactly zero, rows and columns of zeros
        A[:, :25] = 0.0
        Bm[25:, ::2] = 0.0
        A[7], Bm[:, 9] = 0.0, 0.0
    else:
        A, Bm = A * 2.0 ** rng.integers(-60, 60, (n, n)), Bm * 2.0 ** rng.integers(-60, 60, (n, n))
    for t in ORDERS:
        check(one_block(cuda_ctx, n, n, [(A, Bm)], [1.0], [t]), [(A, Bm)], [1.0])


def test_graded_wide_tiles(cuda_ctx):
    """The same in 32 x 32 tiles: many blocks, several chunks a share."""
    rng = np.random.default_rng(12)
    outs, terms, abuf, bbuf, pos = [], [], [], [], []
    ao = bo = co = 0
    for i in range(40):
        M, Nn, K = int(rng.integers(20, 90)), int(rng.integers(20, 90)), int(rng.integers(20, 300))
        A, Bm = graded(rng, M, Nn, K, [0, 1, 3, 10, 30][i % 5])
        a, lda = stored(A, i & 1, 0)
        b, ldb = stored(Bm, i >> 1 & 1, 0)
        terms.append([0, ao, lda, i & 1, 2, bo, ldb, i >> 1 & 1, K])
        outs.append([1, co, M, M, Nn, 0, 1])
        abuf.append(a)
        bbuf.append(b)
        pos.append((co, M, Nn, A, Bm))
        ao, bo, co = ao + a.size, bo + b.size, co + M * Nn
    got = run_program(cuda_ctx, [np.concatenate(abuf), np.full(co, np.nan), np.concatenate(bbuf)], outs, terms,
                      np.ones(len(terms)))
    for c, M, Nn, A, Bm in pos:
        check(got[c:c + M * Nn].reshape(M, Nn, order="F"), [(A, Bm)], [1.0])


@pytest.mark.parametrize("first", [-126, 126, 1])
def test_largest_digit_sums(cuda_ctx, first):
    """Every digit of every entry -128 (or 127), K = 80: level sums of up to 8 * 2^14 * 80, which FP32 holds."""
    low = -128 if first < 0 else 127
    x = first * 2.0 ** -7 + sum(low * 2.0 ** -(7 + 8 * i) for i in range(1, 6))
    for K in (16, 80, 160):
        A, Bm = np.full((20, K), x), np.full((K, 10), x * 2.0 ** 5)
        check(one_block(cuda_ctx, 20, 10, [(A, Bm)], [1.0], [(0, 0)]), [(A, Bm)], [1.0])


def test_integers_are_exact(cuda_ctx):
    rng = np.random.default_rng(13)
    A, Bm = rng.integers(-2 ** 20, 2 ** 20, (37, 75)), rng.integers(-2 ** 20, 2 ** 20, (75, 41))
    got = one_block(cuda_ctx, 37, 41, [(A.astype(float), Bm.astype(float))], [1.0], [(1, 1)])
    assert np.array_equal(got, (A @ Bm).astype(float))


def test_first_digits_at_their_edge(cuda_ctx):
    """Largest entries from just below 127 / 128 of a power of two up to it."""
    x = 1.0 - np.concatenate([2.0 ** -np.arange(5.0, 54.0), 2.0 ** -7 + np.arange(-4.0, 5.0) * 2.0 ** -53])
    for s in (1.0, -1.0):
        A, Bm = np.outer(s * x, [1.0, 0.3, 0.2]), np.array([[0.4, 1.0], [1.0, -0.99609375], [0.7, 0.996]])
        check(one_block(cuda_ctx, len(x), 2, [(A, Bm)], [1.0], [(0, 0)]), [(A, Bm)], [1.0])
