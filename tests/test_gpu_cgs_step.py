"""The cooperative CGS2 step through the Lanczos and GMRES entry points at vector lengths where its work
split changes: one block, a few rows past a block, blocks of 64 rows up to one per SM, more than 311,296
rows (the four-launch form), and bases from 2 to 126 columns.

Operators are diagonal, so the lowest eigenpair is known; the bounds are the solver's own: an eigenvalue
within tol of a symmetric operator's and a solution with |r| <= tol |b|, both times what FP64 sums of n
terms add."""
import numpy as np
import pytest

from imps_cpp_tools_gb300 import ops

pytestmark = pytest.mark.gpu


def diagonal(ctx, d):
    """in_ptr, out_ptr -> out = d * in on the context's stream."""
    import torch
    n = d.numel()

    class Holder:  # a raw device pointer as a tensor
        def __init__(self, ptr):
            self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (ptr, False), "version": 3}

    def apply(pin, pout):
        torch.mul(d, torch.as_tensor(Holder(pin), device="cuda"), out=torch.as_tensor(Holder(pout), device="cuda"))
    return apply


@pytest.mark.parametrize("n,ncv", [(5, 4), (63, 20), (64, 20), (65, 33), (129, 64), (1712, 126), (9728, 40), (9729, 126),
                                   (24368, 17), (48066, 126), (150276, 64), (311296, 20), (311297, 20)])
def test_lanczos_lengths(cuda_ctx, n, ncv):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(n)
    d = torch.linspace(0.0, 1.0, n, dtype=torch.float64, device="cuda") + 1.0
    at = n // 3
    d[at] = -1.0  # the wanted pair, well separated
    x = torch.randn(n, generator=gen, dtype=torch.float64, device="cuda")
    with torch.cuda.stream(torch.cuda.current_stream()):
        vals, _, conv = ops.eigs_rs_op(cuda_ctx, n, diagonal(cuda_ctx, d), x, tol=1e-12, ncv=ncv)
    torch.cuda.synchronize()
    assert conv and abs(vals[0] + 1.0) <= 1e-12 + 1e-15 * np.sqrt(n)
    # eigenvector error <= residual / gap (2)
    v = x.cpu().numpy()
    assert abs(np.linalg.norm(v) - 1.0) <= 1e-14 * np.sqrt(n)
    v[at] = 0.0
    assert np.linalg.norm(v) <= 1e-12 + 1e-14 * np.sqrt(n)
