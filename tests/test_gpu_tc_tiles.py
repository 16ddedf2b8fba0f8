"""The split-BF16 engine at the edges of its tiles: rows around the 8-row groups in which A is packed and the
128-row tile, columns around the 16-wide steps and the 128-column tile, K around the 16-wide steps and the two
of a pipeline stage, one and several terms, plain and accumulated output; values that leave FP32's normal range.

Bound, derived: an operand's three BF16 terms carry 24 bits and the dropped products are below 2^-23, with the
coefficient's rounding below 2^-21 of |a| |b| together; each of the 6 K additions in FP32 truncates by 2^-23 of
a partial sum of at most 1.01 sum |a| |b|."""
import ctypes as C

import numpy as np
import pytest

from imps_cpp_tools_gb300 import _native as N
from imps_cpp_tools_gb300 import blocks as B
from tests.test_gpu_split_gemm import dev, stored

pytestmark = pytest.mark.gpu


def run(ctx, M, Nn, mats, alphas, trans, accumulate):
    abuf, bbuf, terms, ao, bo = [], [], [], 0, 0
    for (A, Bm), (ta, tb) in zip(mats, trans):
        a, lda = stored(A, ta, 1)
        b, ldb = stored(Bm, tb, 0)
        terms.append([0, ao, lda, ta, 2, bo, ldb, tb, A.shape[1]])
        abuf.append(a)
        bbuf.append(b)
        ao, bo = ao + a.size, bo + b.size
    out = np.full((M + 1) * Nn, 3.25)
    bufs = [np.concatenate(abuf), out, np.concatenate(bbuf)]
    sizes, nouts = np.array([len(b) for b in bufs], np.int64), np.array([1], np.int32)
    o = np.array([[1, 0, M + 1, M, Nn, accumulate, len(mats)]], np.int64)
    t, al = np.array(terms, np.int64), np.array(alphas, np.float64)
    h = C.c_void_p()
    N.call("imps_plan_program", ctx.handle, 3, sizes.ctypes.data_as(N.P_i64), 1, nouts.ctypes.data_as(N.P_i32),
           o.ctypes.data_as(N.P_i64), t.ctypes.data_as(N.P_i64), al.ctypes.data_as(N.P_dbl), C.byref(h))
    plan = B.Plan(ctx, h, "program")
    d = [dev(b) for b in bufs]
    for i, x in enumerate(d):
        plan.bind(i, x)
    plan.set_precision(N.PREC_BF16X6)
    plan.run()
    ctx.synchronize()
    return d[1].cpu().numpy().reshape(M + 1, Nn, order="F")


@pytest.mark.parametrize("accumulate", [0, 1])
@pytest.mark.parametrize("M,Nn,ks", [(1, 1, [1]), (7, 15, [16]), (8, 16, [17]), (9, 17, [33, 5]), (64, 33, [48, 15, 64]),
                                     (82, 82, [82] * 6), (127, 129, [31]), (128, 128, [64, 1]), (129, 127, [100]),
                                     (136, 250, [32, 130])])
def test_tile_edges(cuda_ctx, M, Nn, ks, accumulate):
    rng = np.random.default_rng(M * 1000 + Nn)
    mats = [(rng.standard_normal((M, k)), rng.standard_normal((k, Nn))) for k in ks]
    alphas = [1.0, -0.5, 1.7, 0.3, 2.0, -1.1][:len(ks)]
    trans = [(i & 1, (i >> 1) & 1) for i in range(len(ks))]
    got = run(cuda_ctx, M, Nn, mats, alphas, trans, accumulate)
    ref = sum(al * (a @ b) for (a, b), al in zip(mats, alphas)) + 3.25 * accumulate
    mag = sum(abs(al) * (abs(a) @ abs(b)) for (a, b), al in zip(mats, alphas)) + 3.25 * accumulate
    bound = (2.0 ** -21 + 6.1 * sum((k + 15) // 16 * 16 for k in ks) * 2.0 ** -23) * mag
    assert (np.abs(got[:M] - ref) <= bound).all()
    assert (got[M] == 3.25).all()  # past the block


def test_values_written(cuda_ctx):
    """Sums that are zero, denormal in FP32, infinite or not a number come out as their FP32 value."""
    a = np.zeros((9, 4))
    a[:, 0] = [0.0, 1.0, -1.0, 2.0 ** -130, 2.0 ** -140, np.inf, -np.inf, np.nan, 3.0]
    b = np.zeros((4, 20))
    b[0] = 1.0
    got = run(cuda_ctx, 9, 20, [(a, b)], [1.0], [(0, 0)], 0)[:9]
    assert (got[:3] == a[:3, :1]).all() and (got[8] == 3.0).all()
    assert (np.abs(got[3:5] - a[3:5, :1]) <= 2.0 ** -126).all()
    assert not np.isfinite(got[5:8]).any()
