"""Thick restarts of the Lanczos solve, whose basis the grouped GEMM rotates: one and several column tiles (ncv / 2
kept vectors) and K chunks (ncv), a row count that is no multiple of a tile.
The kept basis has to stay orthonormal and span the Ritz vectors, or the next cycles' projected matrix is wrong:
the returned pair has to satisfy the eigenvalue equation to 1e-10 of the operator's norm (the solve stops at
1e-12 of the eigenvalue) and agree with the solve that rotates few vectors to 1e-10."""
import numpy as np
import pytest

from imps_cpp_tools_gb300 import ops
from tests import imps_testlib as T
from tests.test_gpu_parity import _hac_setup, dev, host

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def problem(cuda_ctx):
    model, dims0, _ = T.workload_dims("xxz_d64")
    p = T.hac_problem(model, dims0, seed=5)
    plan, lac = _hac_setup(cuda_ctx, p)
    x0 = p["rng"].standard_normal(lac.nelem)
    x = dev(x0)
    ev, napp, conv = ops.eigs_rs(plan, x, 1e-12, 20)
    assert conv and napp > 20
    return plan, lac.nelem, x0, ev


@pytest.mark.parametrize("ncv", [31, 32, 33, 64, 66, 67, 126])
def test_restarted_lanczos(problem, ncv):
    plan, n, x0, ref = problem
    x, y = dev(x0), dev(np.zeros(n))
    ev, napp, conv = ops.eigs_rs(plan, x, 1e-12, ncv)
    assert conv
    ops.ApplyHAvec(plan, x, y)
    v, hv = host(x), host(y)
    assert abs(np.linalg.norm(v) - 1.0) < 1e-12
    scale = max(abs(ev), np.linalg.norm(hv))
    assert np.linalg.norm(hv - ev * v) <= 1e-10 * scale
    assert abs(ev - ref) <= 1e-10 * abs(ref)


@pytest.mark.parametrize("ncv", [32, 64, 126])
def test_many_restarts(problem, ncv):
    """An unreachable tolerance over restart cycles: the Ritz value stays within rounding of the ground state."""
    plan, n, x0, ref = problem
    x = dev(x0)
    ev, napp, _ = ops.eigs_rs(plan, x, 1e-30, ncv, 6)
    assert napp > ncv  # at least one restart
    assert abs(ev - ref) <= 1e-10 * abs(ref)
