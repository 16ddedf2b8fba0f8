"""imps_invert_e_fac takes the real and the imaginary part through each transfer-matrix stage in one launch,
with their own scratch and split-K workspace.  At sizes with 16- and 32-wide tiles, one or several shares,
the solution has to satisfy y - fac T(y) = x with T applied to one part at a time: GMRES stops at 1e-12 of
|x| by its own estimate, and a tenfold of that is allowed for."""
import numpy as np
import pytest

from imps_cpp_tools_gb300 import blocks as B
from imps_cpp_tools_gb300 import configs, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("direction", [0, 1])
@pytest.mark.parametrize("D", [9, 70, 400])
@pytest.mark.parametrize("tuned", [False, True])
def test_solves_its_equation(cuda_ctx, D, direction, tuned):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(D)
    rand = lambda n: torch.randn(n, generator=gen, dtype=torch.float64, device="cuda")
    bond = configs.xxz_bond_dims(D, 3, 3.0)
    I2K = [(1,), (-1,)]
    nxt = {}
    for (q,), m in bond.items():
        for k in I2K:
            nxt.setdefault((q + k[0],), 0)
    for q in nxt:
        nxt[q] = max(1, sum(bond.get((q[0] + s,), 0) for s in (1, -1)) // 2)
    lays = []
    for left, right in ((bond, nxt), (nxt, bond)):
        lays.append(B.Layout([(s, l, (l[0] + k[0],), left[l], right[(l[0] + k[0],)])
                              for s, k in enumerate(I2K) for l in sorted(left) if (l[0] + k[0],) in right], 1))
    lay = B.Layout([(0, q, q, m, m) for q, m in sorted(bond.items())], 1)
    plan = B.plan_tm_mixed(cuda_ctx, lays, lays, direction, lay, lay)
    for k in range(2):
        scale = 0.3 / np.sqrt(D)
        plan.bind(2 + k, scale * rand(lays[k].nelem))
        plan.bind(4 + k, scale * rand(lays[k].nelem))
    if tuned:
        plan.autotune(3)
    n = lay.nelem
    xr, xi, yr, yi = rand(n), rand(n), rand(n), rand(n)
    fac = np.exp(0.8j)
    it, rr, conv = ops.InvertE_fac(plan, xr, xi, fac, yr, yi, 1e-12)
    assert conv and it > 0
    tr, ti = torch.empty_like(yr), torch.empty_like(yi)
    ops.ApplyTM(plan, yr, tr)
    ops.ApplyTM(plan, yi, ti)
    cuda_ctx.synchronize()
    rr = yr - (fac.real * tr - fac.imag * ti) - xr
    ri = yi - (fac.real * ti + fac.imag * tr) - xi
    norm = torch.sqrt(xr.dot(xr) + xi.dot(xi))
    assert torch.sqrt(rr.dot(rr) + ri.dot(ri)) <= 1e-11 * norm
