"""The cooperative CGS2 step through GMRES, whose first pass takes all columns: one block, a few rows past a
block, blocks of 64 rows up to one per SM and more, up to 80 columns; and vectors that lie in the span of the
basis but for rounding, whose norm is summed explicitly.

The transfer matrix T(X) = O^T X O of an orthogonal O (two tensors O / sqrt(2)) is unitary, with O's
eigenvalues' products as its own, so (1 - f T) y = x has a closed form, |(1 - f T)^-1| <= 1 / (1 - f), and for
f = 0.95 GMRES needs its whole Krylov space.  Bound: |y - exact| <= tol |x| / (1 - f), as |r| <= tol |x|, doubled
for the residual's own rounding."""
import numpy as np
import pytest

from imps_cpp_tools_gb300 import blocks as B
from imps_cpp_tools_gb300 import ops

pytestmark = pytest.mark.gpu
TOL = 1e-11


def dev(a):
    import torch
    return torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


class Problem:
    def __init__(self, ctx, m):
        rng = np.random.default_rng(m)
        self.m, self.rng = m, rng
        O = np.linalg.qr(rng.standard_normal((m, m)))[0]
        la = B.Layout([(s, (0,), (0,), m, m) for s in (0, 1)], 1)
        lay = B.Layout([(0, (0,), (0,), m, m)], 1)
        A = (O / np.sqrt(2.0)).reshape(-1, order="F")
        self.plan = B.plan_tm_mixed(ctx, [la], [la], 0, lay, lay)
        self.keep = dev(np.concatenate([A, A]))
        self.plan.bind(2, self.keep)
        self.plan.bind(3, self.keep)
        d, self.W = np.linalg.eig(O)  # O is normal with distinct eigenvalues: W is unitary
        self.dd = d[:, None] * d[None, :]

    def coefficients(self, X):
        return self.W.T @ X @ self.W

    def matrix(self, Z):
        return self.W.conj() @ Z @ self.W.conj().T

    def solve(self, X, fac):
        re, im = (dev(p.reshape(-1, order="F")) for p in (X.real, X.imag))
        y = [dev(np.zeros(self.m * self.m)) for _ in range(2)]
        it, rel, conv = ops.InvertE_fac(self.plan, re, im, complex(fac), y[0], y[1], TOL)
        Y = sum(c * p.cpu().numpy().reshape(self.m, self.m, order="F") for c, p in zip((1.0, 1j), y))
        exact = self.matrix(self.coefficients(X) / (1.0 - fac * self.dd))
        assert conv and np.isfinite(Y).all()
        assert np.linalg.norm(Y - exact) <= 2 * TOL * np.linalg.norm(X) / (1.0 - abs(fac))
        return it


# 2 m^2 rows: 50, 72, 128, 162, 1,058, 9,522, 9,800, 20,000, 45,000
@pytest.mark.parametrize("m", [5, 6, 8, 9, 23, 69, 70, 100, 150])
@pytest.mark.parametrize("fac", [0.95, 0.9 * np.exp(0.7j)])
def test_lengths(cuda_ctx, m, fac):
    p = Problem(cuda_ctx, m)
    X = p.rng.standard_normal((m, m)) + 1j * p.rng.standard_normal((m, m))
    it = p.solve(X, fac)
    if m >= 23:
        assert it > 64  # more than 64 columns of the basis


@pytest.mark.parametrize("m", [9, 70])
@pytest.mark.parametrize("k", [1, 2, 5, 6])
def test_span(cuda_ctx, m, k):
    """x in an invariant subspace of dimension 2 k (real and imaginary parts): the steps past it, up to the next
    check, orthogonalise what is rounding alone."""
    p = Problem(cuda_ctx, m)
    Z = np.zeros((m, m), complex)
    for i in range(k):
        Z[i, (2 * i) % m] = 1.0 + 0.5j * i
    p.solve(p.matrix(Z), 0.6)
