"""The FP64 grouped GEMM at the sizes where its tiling and operand splitting can go wrong: block edges
around the 16- and 32-row tiles and 8-column strips, K around the 16-wide steps and the 80-wide chunks,
both storage orders of both operands, padded leading dimensions, coefficients, accumulation, empty
sums; and operands it must not split (not finite, or scales near the ends of the FP64 range).

Bounds, derived: per term and output, digits dropped and rounded off are below 2^-54 of the product of
the row's and the column's power-of-two scales, each at most twice the largest entry, i.e. 2^-52 of the
product of the largest entries, for each of the K products; every FP64 operation of the accumulation
rounds by 2^-53 of a partial sum of magnitudes (a few per term, doubled for the reference's own)."""
import ctypes as C

import numpy as np
import pytest

from imps_cpp_tools_gb300 import _native as N
from imps_cpp_tools_gb300 import blocks as B

pytestmark = pytest.mark.gpu


def dev(a):
    import torch
    return torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def run_program(ctx, bufs, outs, terms, alphas):
    nouts = np.array([len(outs)], np.int32)
    sizes = np.array([len(b) for b in bufs], np.int64)
    o, t, al = np.array(outs, np.int64), np.array(terms, np.int64), np.array(alphas, np.float64)
    h = C.c_void_p()
    N.call("imps_plan_program", ctx.handle, len(bufs), sizes.ctypes.data_as(N.P_i64), 1, nouts.ctypes.data_as(N.P_i32),
           o.ctypes.data_as(N.P_i64), t.ctypes.data_as(N.P_i64), al.ctypes.data_as(N.P_dbl), C.byref(h))
    plan = B.Plan(ctx, h, "program")
    d = [dev(b) for b in bufs]
    for i, x in enumerate(d):
        plan.bind(i, x)
    plan.run()
    ctx.synchronize()
    return d[1].cpu().numpy()


def stored(M, trans, pad):
    """op()^-1(M) column-major with `pad` rows more than needed: (flat buffer, leading dimension)."""
    S = M.T if trans else M
    buf = np.full((S.shape[0] + pad, max(S.shape[1], 1)), 7.5)
    buf[:S.shape[0], :S.shape[1]] = S
    return buf.reshape(-1, order="F"), S.shape[0] + pad


def one_block(ctx, M, Nn, mats, alphas, trans, pad=0, accumulate=None):
    """sum_t alpha_t A_t B_t into one M x Nn block; mats: list of (A, B)."""
    abuf, bbuf, terms = [], [], []
    ao = bo = 0
    for (A, Bm), (ta, tb) in zip(mats, trans):
        a, lda = stored(A, ta, pad)
        b, ldb = stored(Bm, tb, pad)
        terms.append([0, ao, lda, ta, 2, bo, ldb, tb, A.shape[1]])
        abuf.append(a)
        bbuf.append(b)
        ao += a.size
        bo += b.size
    out = np.full((M + pad) * Nn, 3.25) if accumulate is None else accumulate.copy()
    cat = lambda x: np.concatenate(x) if x else np.zeros(1)
    got = run_program(ctx, [cat(abuf), out, cat(bbuf)], [[1, 0, M + pad, M, Nn, int(accumulate is not None), len(mats)]],
                      terms if terms else np.zeros((0, 9)), alphas)
    return got.reshape(M + pad, Nn, order="F")


def check(got, M, mats, alphas, start=0.0):
    ref = np.zeros(got[:M].shape, np.longdouble) + start
    bound = np.abs(ref) * 2.0 ** -52
    for (A, Bm), al in zip(mats, alphas):
        a, b = A.astype(np.longdouble), Bm.astype(np.longdouble)
        ref = ref + al * (a @ b)
        if A.shape[1]:
            ra, cb = np.abs(A).max(1)[:, None], np.abs(Bm).max(0)[None, :]
            bound = bound + abs(al) * (A.shape[1] * 2.0 ** -52 * ra * cb + (8 + len(mats)) * 2.0 ** -53 * (np.abs(A) @ np.abs(Bm)))
    err = np.abs(got[:M] - ref)
    assert np.isfinite(got[:M]).all()
    assert (err <= bound).all(), float((err / np.maximum(bound, 1e-300)).max())


@pytest.mark.parametrize("M,Nn", [(1, 1), (8, 9), (15, 17), (16, 8), (17, 33), (31, 7), (32, 32), (33, 31), (68, 68), (82, 1),
                                  (1, 82), (113, 40)])
@pytest.mark.parametrize("K", [1, 15, 16, 17, 63, 80, 81, 160, 161, 300])
def test_edges(cuda_ctx, M, Nn, K):
    rng = np.random.default_rng(M * 1000 + Nn * 10 + K)
    # three terms of different length, the rows and columns over many binades
    ks = [K, max(1, K // 3), 2]
    mats = [(rng.standard_normal((M, k)) * 2.0 ** rng.integers(-30, 30, (M, 1)),
             rng.standard_normal((k, Nn)) * 2.0 ** rng.integers(-30, 30, (1, Nn))) for k in ks]
    alphas = [1.0, -0.75, 3.0]
    for trans in ([(0, 0)] * 3, [(1, 0), (0, 1), (1, 1)], [(0, 1), (1, 1), (1, 0)]):
        check(one_block(cuda_ctx, M, Nn, mats, alphas, trans, pad=3), M, mats, alphas)


def test_many_blocks_share_chunks(cuda_ctx):
    """Enough blocks for 32 x 32 tiles, with more K chunks than shares, shares cut inside a term."""
    rng = np.random.default_rng(5)
    outs, terms, abuf, bbuf, all_mats, pos = [], [], [], [], [], []
    ao = bo = co = 0
    for i in range(40):
        M, Nn = int(rng.integers(20, 90)), int(rng.integers(20, 90))
        ks = [int(k) for k in rng.integers(1, 400, int(rng.integers(1, 9)))]
        mats = [(rng.standard_normal((M, k)), rng.standard_normal((k, Nn))) for k in ks]
        for A, Bm in mats:
            a, lda = stored(A, 0, 0)
            b, ldb = stored(Bm, 1, 0)
            terms.append([0, ao, lda, 0, 2, bo, ldb, 1, A.shape[1]])
            abuf.append(a)
            bbuf.append(b)
            ao += a.size
            bo += b.size
        outs.append([1, co, M, M, Nn, 0, len(mats)])
        pos.append((co, M, Nn))
        co += M * Nn
        all_mats.append(mats)
    bufs = [np.concatenate(abuf), np.full(co, np.nan), np.concatenate(bbuf)]
    got = run_program(cuda_ctx, bufs, outs, terms, np.ones(len(terms)))
    for (c, M, Nn), mats in zip(pos, all_mats):
        check(got[c:c + M * Nn].reshape(M, Nn, order="F"), M, mats, [1.0] * len(mats))
    again = run_program(cuda_ctx, bufs, outs, terms, np.ones(len(terms)))
    assert np.array_equal(got, again)  # the same sums in the same order


def test_accumulate_and_empty(cuda_ctx):
    rng = np.random.default_rng(3)
    A, Bm = rng.standard_normal((20, 30)), rng.standard_normal((30, 12))
    start = rng.standard_normal(20 * 12)
    got = one_block(cuda_ctx, 20, 12, [(A, Bm)], [1.0], [(0, 0)], accumulate=start)
    check(got, 20, [(A, Bm)], [1.0], start.reshape(20, 12, order="F"))
    assert (one_block(cuda_ctx, 20, 12, [], [], []) == 0.0).all()  # no terms
    got = one_block(cuda_ctx, 20, 12, [(np.zeros((20, 0)), np.zeros((0, 12))), (A, Bm)], [1.0, 1.0], [(0, 0)] * 2)
    check(got, 20, [(A, Bm)], [1.0])  # an empty sum before another
    assert (one_block(cuda_ctx, 20, 12, [(A * 0.0, Bm)], [1.0], [(0, 0)]) == 0.0).all()


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_not_finite(cuda_ctx, value):
    rng = np.random.default_rng(4)
    A, Bm, A2, B2 = (rng.standard_normal(s) for s in ((40, 50), (50, 24), (40, 90), (90, 24)))
    A[3, 7] = value
    Bm[11, 5] = value
    got = one_block(cuda_ctx, 40, 24, [(A, Bm), (A2, B2)], [1.0, 1.0], [(0, 0), (1, 0)])
    with np.errstate(invalid="ignore"):
        ref = A @ Bm + A2 @ B2
    bad = ~np.isfinite(ref)
    assert bad.any() and not bad.all()
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    assert np.array_equal(got[bad & ~np.isnan(ref)], ref[bad & ~np.isnan(ref)])
    mag = (np.abs(np.where(np.isfinite(A), A, 0)) @ np.abs(np.where(np.isfinite(Bm), Bm, 0)) + np.abs(A2) @ np.abs(B2))
    assert (np.abs(got - ref)[~bad] <= 200 * 2.0 ** -52 * mag[~bad]).all()


@pytest.mark.parametrize("sa,sb", [(2.0 ** -1030, 2.0 ** 900), (2.0 ** 900, 2.0 ** -900), (2.0 ** -600, 2.0 ** -440),
                                   (2.0 ** 600, 2.0 ** 400), (2.0 ** -420, 2.0 ** 470), (5e-324, 1.0)])
def test_extreme_scales(cuda_ctx, sa, sb):
    """Rows near the ends of the FP64 range, subnormal ones among them: the FP64 results."""
    rng = np.random.default_rng(6)
    A, Bm = np.round(rng.standard_normal((18, 40)) * 1024) * sa, rng.standard_normal((40, 20)) * sb
    got = one_block(cuda_ctx, 18, 20, [(A, Bm)], [1.0], [(0, 0)])
    ref = A.astype(np.longdouble) @ Bm.astype(np.longdouble)
    mag = np.abs(A).astype(np.longdouble) @ np.abs(Bm).astype(np.longdouble)
    tiny = np.longdouble(5e-324)
    # one rounding per multiply-add, in units of the last place or of the smallest subnormal
    assert (np.abs(got - ref) <= 42 * (np.longdouble(2.0) ** -53 * mag + tiny) + 42 * 2.0 ** -52 *
            np.abs(A).max(1)[:, None].astype(np.longdouble) * np.abs(Bm).max(0)[None, :].astype(np.longdouble)).all()
    if abs(sa * sb) > 0:
        assert (got != 0).any()


@pytest.mark.parametrize("n", [1, 7, 16, 33, 82])
def test_selection_is_exact(cuda_ctx, n):
    """A product with an identity, a permutation or a diagonal keeps every entry's own 53 bits."""
    rng = np.random.default_rng(7)
    X = rng.standard_normal((n, n)) * 2.0 ** rng.integers(-300, 100, (n, n))
    P, D = np.eye(n)[rng.permutation(n)], np.diag(2.0 ** rng.integers(-5, 5, n))
    for S in (np.eye(n), P, D, -P):
        assert np.array_equal(one_block(cuda_ctx, n, n, [(X, S)], [1.0], [(0, 1)]), X @ S)
        assert np.array_equal(one_block(cuda_ctx, n, n, [(S, X)], [1.0], [(1, 0)]), S @ X)
