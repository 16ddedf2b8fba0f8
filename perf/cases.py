"""The framework's hot path as cases to time: what a VUMPS or excitation program calls in earnest.

A case names one public entry point ("op"), a model ("xxz": spin-1/2 XXZ chain with U(1) charges;
"fhub": Fermi-Hubbard chain with U(1) x U(1) charges), the total bond dimension D, spread over
charge sectors as the package's own workloads spread it, and the entry point's options.  Inputs are
seeded: Gaussian blocks, made isometric where the path only ever meets isometries.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from imps_cpp_tools_gb300 import _native as N
from imps_cpp_tools_gb300 import blocks as B
from imps_cpp_tools_gb300 import configs, models, ops

F64 = torch.float64
PARAMS = {"xxz": {"J": 1.0, "Delta": -1.0}, "fhub": {"t": 1.0, "U": 4.0}}


def listed():
    return [
        # one H_AC apply of the smallest documented chain: launch and latency bound, as in quick studies
        {"name": "hac xxz 64", "op": "hac", "model": "xxz", "D": 64},
        # the H_AC apply that every Lanczos step of a production sweep makes
        {"name": "hac xxz 512", "op": "hac", "model": "xxz", "D": 512},
        # the same at the largest documented size, d = 4 and 60 uneven sectors
        {"name": "hac fhub 1024", "op": "hac", "model": "fhub", "D": 1024},
        # the split-BF16 option of that apply
        {"name": "hac mixed fhub 1024", "op": "hac", "model": "fhub", "D": 1024, "precision": "bf16x6"},
        # the centre-matrix apply of the H_C eigensolves, an odd total dimension
        {"name": "hc xxz 389", "op": "hc", "model": "xxz", "D": 389},
        # a unit-cell transfer matrix from the left (environments, observables)
        {"name": "tm left xxz 512", "op": "tm", "model": "xxz", "D": 512, "dir": "l"},
        # the projected transfer matrix from the right, which the GMRES iterates on
        {"name": "tm proj right fhub 1024", "op": "tmproj", "model": "fhub", "D": 1024, "dir": "r"},
        # an environment solve, twice per site update
        {"name": "env left xxz 512", "op": "env", "model": "xxz", "D": 512, "dir": "l"},
        # an H_AC ground state, the larger part of a site update, with the driver's basis and tolerance
        {"name": "lanczos xxz 512", "op": "lanczos", "model": "xxz", "D": 512},
        # the QR form of the A_L / A_R update (near convergence)
        {"name": "qr fhub 1024", "op": "qr", "model": "fhub", "D": 1024},
        # the polar form of the A_L / A_R update (far from convergence)
        {"name": "polar xxz 512", "op": "polar", "model": "xxz", "D": 512},
        # one momentum's environment solve of the excitation ansatz: complex, mixed transfer matrix
        {"name": "momentum xxz 256", "op": "momentum", "model": "xxz", "D": 256, "dir": "r"},
    ]


def draw(rng):
    op = rng.choice(["hac", "hac", "hac mixed", "hc", "tm", "tmproj", "env", "lanczos", "qr", "polar", "momentum"])
    model = rng.choice(["xxz", "xxz", "fhub"])
    top = {"lanczos": 512, "momentum": 256, "env": 512}.get(op, 1024)
    lo = 32 if model == "xxz" else 64
    D = int(round(math.exp(rng.uniform(math.log(lo), math.log(top)))))
    case = {"op": op.split()[0], "model": model, "D": D}
    if op == "hac mixed":
        case["precision"] = "bf16x6"
    if op in ("tm", "tmproj", "env", "momentum"):
        case["dir"] = rng.choice(["l", "r"])
    return case


# ---------------------------------------------------------------------------------- sector tables

def bond_dims(model, D):
    """Sectors of bond 0: as many and as spread out as the package's workloads of about this D have."""
    if model == "xxz":
        qmax = max(2, round(2 * math.log2(D) - 8))
        return configs.xxz_bond_dims(D, qmax, qmax * qmax / 5.5)
    return configs.hubbard_bond_dims(D, max(12, round(10 * math.log2(D) - 40)))


class Structure:
    """Two-site unit cell: site n maps bond n to bond 1 - n."""

    def __init__(self, case):
        self.d, self.I2K, h = models.build_model(case["model"], **PARAMS[case["model"]])
        self.hnnz = models.h_nonzeros(h)
        self.bonds = models.make_dims(bond_dims(case["model"], case["D"]), 2, self.I2K)
        self.start, self.dim = [], []
        for b in self.bonds:
            at, pos = {}, 0
            for q in sorted(b):
                at[q] = pos
                pos += b[q]
            self.start.append(at)
            self.dim.append(pos)

    def mps(self, n):
        """Blocks (s, left charge, right charge) of a tensor on site n, in the flat buffer's order."""
        l, r = self.bonds[n], self.bonds[1 - n]
        plus = lambda q, s: tuple(a + b for a, b in zip(q, self.I2K[s]))
        return [(s, q, plus(q, s)) for s in range(self.d) for q in sorted(l) if plus(q, s) in r]

    def mixed(self, b):
        """Charges (q, q + 2 quanta) of a block matrix on bond b that raises the charge."""
        up = (2,) + (0,) * (len(self.I2K[0]) - 1)
        plus = lambda q: tuple(x + y for x, y in zip(q, up))
        return [(q, plus(q)) for q in sorted(self.bonds[b]) if plus(q) in self.bonds[b]]

    def layout(self, n):
        return B.Layout.mps(self.I2K, self.bonds[n], self.bonds[1 - n])

    def mps_size(self, n):
        return sum(self.bonds[n][l] * self.bonds[1 - n][r] for _, l, r in self.mps(n))

    def bd_size(self, b):
        return sum(m * m for m in self.bonds[b].values())


def gauss(gen, *shape):
    return torch.randn(*shape, generator=gen, dtype=F64, device="cuda")


def generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 31))


def split_mps(S, n, v):
    """The blocks of a flat site tensor, as matrices {(s, ql): (qr, M)}."""
    out, o = {}, 0
    for s, l, r in S.mps(n):
        a, b = S.bonds[n][l], S.bonds[1 - n][r]
        out[(s, l)] = (r, v[o:o + a * b].reshape(b, a).T)
        o += a * b
    return out


def flat(mats):
    return torch.cat([m.T.reshape(-1) for m in mats]).contiguous()


def isometry(S, n, gen, side):
    """A random left- (side "l") or right-isometric site tensor, flat."""
    M = split_mps(S, n, gauss(gen, S.mps_size(n)))
    group = {}
    for (s, l), (r, m) in M.items():
        group.setdefault(r if side == "l" else l, []).append((s, l))
    for keys in group.values():
        stack = torch.cat([M[k][1] if side == "l" else M[k][1].T for k in keys])
        q, o = torch.linalg.qr(stack)[0], 0
        for k in keys:
            rows = M[k][1].shape[0 if side == "l" else 1]
            part = q[o:o + rows]
            M[k] = (M[k][0], part if side == "l" else part.T)
            o += rows
    return flat([M[(s, l)][1] for s, l, _ in S.mps(n)])


def symmetric(S, b, gen):
    return flat([0.5 * (m + m.T) for m in (gauss(gen, x, x) for _, x in sorted(S.bonds[b].items()))])


def density(S, b, gen):
    """C C^T of unit trace: a right (left) fixed point's guess."""
    ms = [m @ m.T for m in (gauss(gen, x, x) for _, x in sorted(S.bonds[b].items()))]
    v = flat(ms)
    return v / sum(torch.trace(m) for m in ms)


def eye(S, b):
    return flat([torch.eye(x, dtype=F64, device="cuda") for _, x in sorted(S.bonds[b].items())])


def graded(S, n, gen, side):
    """A site tensor Q P with Q isometric and P positive, its singular values over four decades per
    sector: what the polar step meets, A_C C^T."""
    M = split_mps(S, n, isometry(S, n, gen, side))
    bond = S.bonds[1 - n] if side == "l" else S.bonds[n]
    P = {}
    for q in sorted(bond):
        m = bond[q]
        o = torch.linalg.qr(gauss(gen, m, m))[0]
        P[q] = (o * torch.logspace(0, -4, m, dtype=F64, device="cuda")) @ o.T
    return flat([M[(s, l)][1] @ P[r] if side == "l" else P[l] @ M[(s, l)][1] for s, l, r in S.mps(n)])


def inputs(case, seed):
    """The seeded operands by name, as flat buffers."""
    S, gen = Structure(case), generator(seed)
    op = case["op"]
    x = {}
    if op in ("hac", "lanczos"):
        # A_C on site 0, A_L and A_R on site 1 to its left and right
        x["AL"], x["AR"] = isometry(S, 1, gen, "l"), isometry(S, 1, gen, "r")
        x["EHL"], x["EHR"] = symmetric(S, 0, gen), symmetric(S, 1, gen)
        x["v"] = gauss(gen, S.mps_size(0))
    elif op == "hc":
        x["AL"], x["AR"] = isometry(S, 1, gen, "l"), isometry(S, 0, gen, "r")
        x["EHL"], x["EHR"], x["v"] = symmetric(S, 0, gen), symmetric(S, 0, gen), gauss(gen, S.bd_size(0))
    elif op in ("tm", "tmproj", "env"):
        x["A0"], x["A1"] = isometry(S, 0, gen, case["dir"]), isometry(S, 1, gen, case["dir"])
        x["v"], x["rho"] = symmetric(S, 0, gen), density(S, 0, gen)
    elif op == "qr":
        x["v"], x["c"] = gauss(gen, S.mps_size(0)), gauss(gen, S.bd_size(1))
    elif op == "polar":
        x["l"], x["r"] = graded(S, 0, gen, "l"), graded(S, 0, gen, "r")
    elif op == "momentum":
        for n in (0, 1):
            x["A%d" % n], x["B%d" % n] = isometry(S, n, gen, "l"), isometry(S, n, gen, "r")
        n = sum(S.bonds[0][a] * S.bonds[0][b] for a, b in S.mixed(0))
        x["re"], x["im"] = gauss(gen, n), gauss(gen, n)
        x["p"] = math.pi * (0.1 + 0.8 * torch.rand(1, generator=gen, dtype=F64, device="cuda").item())
    return S, x


# ------------------------------------------------------------------------------------ the program

def prepare(case, seed):
    S, x = inputs(case, seed)
    ctx = B.Context(0, torch.cuda.current_stream())
    op, st = case["op"], {"ctx": ctx, "x": x, "op": case["op"]}
    new = lambda n: torch.zeros(max(n, 1), dtype=F64, device="cuda")
    bd = [B.Layout.blockdiag(b) for b in S.bonds]
    if op in ("hac", "lanczos"):
        la = S.layout(1)
        reduced = []
        for side, A in ((0, x["AL"]), (1, x["AR"])):
            p = B.plan_redop(ctx, la, S.d, S.hnnz, side)
            lay = p.derived(0)
            H = new(lay.nelem)
            p.bind(0, A)
            p.bind(1, H)
            p.run()
            reduced.append((lay, H))
        plan = B.plan_hac(ctx, S.layout(0), bd[0], bd[1], reduced[0][0], reduced[1][0], S.d)
        for k, t in ((2, x["EHL"]), (3, x["EHR"]), (4, reduced[0][1]), (5, reduced[1][1])):
            plan.bind(k, t)
        if case.get("precision") == "bf16x6":
            plan.set_precision(N.PREC_BF16X6)
        plan.prepare()
        st.update(plan=plan, out=new(S.mps_size(0)))
    elif op == "hc":
        plan = B.plan_hc(ctx, bd[0], bd[0], bd[0], S.layout(1), S.layout(0), S.d, S.hnnz)
        for k, t in ((2, x["EHL"]), (3, x["EHR"]), (4, x["AL"]), (5, x["AR"])):
            plan.bind(k, t)
        plan.prepare()
        st.update(plan=plan, out=new(S.bd_size(0)))
    elif op in ("tm", "tmproj", "env"):
        left = case["dir"] == "l"
        plan = B.plan_tm(ctx, [S.layout(0), S.layout(1)], 0 if left else 1, bd[0], bd[0])
        plan.bind(2, x["A0"])
        plan.bind(3, x["A1"])
        one = eye(S, 0)
        # fixed points: the identity on the isometric side, the density on the other
        st.update(plan=plan, out=new(S.bd_size(0)), dir=case["dir"], inner=x["rho"], outer=one,
                  L=one if left else x["rho"], R=x["rho"] if left else one)
    elif op == "qr":
        st.update(dec=B.plan_decomp(ctx, S.layout(0), "l"), decc=B.plan_decomp(ctx, bd[1], "l"),
                  Q=new(S.mps_size(0)), R=new(S.bd_size(1)), P=new(S.bd_size(1)), R2=new(S.bd_size(1)))
    elif op == "polar":
        la = S.layout(0)
        dl, dr = B.plan_decomp(ctx, la, "l"), B.plan_decomp(ctx, la, "r")
        st.update(decs=[dl, dr], U=[new(S.mps_size(0)) for _ in "lr"], V=[new(S.bd_size(1)), new(S.bd_size(0))],
                  sv=[new(dl.nsv), new(dr.nsv)], A=[new(S.mps_size(0)) for _ in "lr"],
                  mul=[B.plan_mps_bd(ctx, la, bd[1], 1), B.plan_mps_bd(ctx, la, bd[0], 0)])
    elif op == "momentum":
        m = S.bonds[0]
        lay = B.Layout([(0, a, b, m[a], m[b]) for a, b in S.mixed(0)], len(S.I2K[0]))
        las = [S.layout(0), S.layout(1)]
        plan = B.plan_tm_mixed(ctx, las, las, 0 if case["dir"] == "l" else 1, lay, lay)
        for k, t in enumerate(("A0", "A1", "B0", "B1")):
            plan.bind(2 + k, x[t])
        st.update(plan=plan, fac=complex(math.cos(x["p"]), math.sin(x["p"])))
    return st


def run(st):
    op, x = st["op"], st["x"]
    if op == "hac":
        return ops.ApplyHAvec(st["plan"], x["v"], st["out"])
    if op == "hc":
        return ops.ApplyHCvec(st["plan"], x["v"], st["out"])
    if op == "tm":
        return ops.ApplyTM(st["plan"], x["v"], st["out"])
    if op == "tmproj":
        return ops.InvEfun_proj(st["plan"], x["v"], st["inner"], st["outer"], st["out"])
    if op == "env":
        y = torch.zeros_like(x["v"])
        ops.InvertE_proj(st["plan"], x["v"], st["L"], st["R"], st["dir"], y, 1e-13)
        return y
    if op == "lanczos":
        # the driver's settings: basis 126, eigensolver tolerance 1e-12 with its margin of ten
        v = x["v"].clone()
        e, _, _ = ops.eigs_rs(st["plan"], v, 1e-13, ncv=126)
        # the side of the start vector: the driver's own rule, the first entry's sign, is that of an
        # outermost sector's rounding here
        return {"energy": e, "vector": v * torch.sign(torch.dot(v, x["v"]))}
    if op == "qr":
        ops.qr(st["dec"], x["v"], st["Q"], st["R"])
        ops.qr(st["decc"], x["c"], st["P"], st["R2"])
        return [st["Q"], st["R"], st["P"], st["R2"]]
    if op == "polar":
        ops.svd_batch(st["decs"], [x["l"], x["r"]], st["U"], st["sv"], st["V"])
        for k in (0, 1):
            p = st["mul"][k]
            p.bind(0, st["U"][k])
            p.bind(1, st["V"][k])
            p.bind(2, st["A"][k])
            p.run()
        return st["A"] + st["sv"]
    y = [torch.zeros_like(x["re"]), torch.zeros_like(x["re"])]
    ops.InvertE_fac(st["plan"], x["re"], x["im"], st["fac"], y[0], y[1], 1e-12)
    return y


# ------------------------------------------------------------------------------ what it has to do

def apply_flops(S, op):
    """Multiply-adds of one apply, twice: the block products that the operator is made of."""
    m, d = S.bonds, S.d
    if op == "hac":
        f = 0
        at = {(s, l): r for s, l, r in S.mps(0)}
        pairs = {(int(r) % d, int(c) % d) for r, c, _ in S.hnnz}
        for s, l, r in S.mps(0):
            a, b = m[0][l], m[1][r]
            f += a * a * b + a * b * b
            for i, j in pairs:
                for (s2, l2), r2 in at.items():
                    if i == s and s2 == j and r2 == r:
                        f += a * m[0][l2] * b
                    if i == s and s2 == j and l2 == l:
                        f += a * m[1][r2] * b
        return 2 * f
    if op == "hc":
        return 2 * sum(2 * (1 + len({(int(r) % d, int(c) % d) for r, c, _ in S.hnnz})) * x ** 3 for x in m[0].values())
    return 2 * sum(m[n][l] * m[1 - n][r] * (m[n][l] + m[1 - n][r]) for n in (0, 1) for _, l, r in S.mps(n))


def work(case):
    S, op = Structure(case), case["op"]
    n0, n1 = S.mps_size(0), S.mps_size(1)
    b0, b1 = S.bd_size(0), S.bd_size(1)
    if op in ("hac", "lanczos"):
        per = apply_flops(S, "hac")
        # the reduced operators have at most d * d blocks for each block of their bond
        bytes_ = 8 * (2 * n0 + (1 + S.d) * (b0 + b1))
        if op == "hac":
            return {"bytes": bytes_, "flops": per}
        k = 100  # steps of a solve, about
        return {"bytes": bytes_ + 8 * n0 * k, "flops": k * per + 4.0 * n0 * k * k / 2}
    if op == "hc":
        return {"bytes": 8 * (4 * b0 + n0 + n1), "flops": apply_flops(S, "hc")}
    if op in ("tm", "tmproj"):
        return {"bytes": 8 * (n0 + n1 + (2 if op == "tm" else 4) * b0), "flops": apply_flops(S, "tm")}
    if op == "env":
        k = 60
        return {"bytes": 8 * (n0 + n1 + 4 * b0 + b0 * k), "flops": k * apply_flops(S, "tm") + 4.0 * b0 * k * k / 2}
    if op == "momentum":
        k, c = 60, sum(S.bonds[0][a] * S.bonds[0][b] for a, b in S.mixed(0))
        return {"bytes": 8 * (2 * (n0 + n1) + 4 * c + 2 * c * k),
                "flops": 2.0 * k * apply_flops(S, "tm") * c / b0 + 8.0 * c * k * k / 2}
    rows = {}
    for s, l, r in S.mps(0):
        rows.setdefault(("l", r), [0, S.bonds[1][r]])[0] += S.bonds[0][l]
        rows.setdefault(("r", l), [0, S.bonds[0][l]])[0] += S.bonds[1][r]
    if op == "qr":
        f = sum(4.0 * a * b * b for (side, _), (a, b) in rows.items() if side == "l") + sum(
            4.0 * x ** 3 for x in S.bonds[1].values())
        return {"bytes": 8 * (2 * n0 + 4 * b1), "flops": f}
    # singular value decomposition of every sector and the product of its two factors
    return {"bytes": 8 * (4 * n0 + b0 + b1), "flops": sum(14.0 * a * b * b + 8.0 * b ** 3 for a, b in rows.values())}


# ------------------------------------------------------------------------------------- exact values

def dense_mps(S, n, v):
    A = torch.zeros(S.d, S.dim[n], S.dim[1 - n], dtype=F64, device="cuda")
    for (s, l), (r, m) in split_mps(S, n, v).items():
        a, b = S.start[n][l], S.start[1 - n][r]
        A[s, a:a + m.shape[0], b:b + m.shape[1]] = m
    return A


def flat_mps(S, n, A):
    a, b = S.start[n], S.start[1 - n]
    return flat([A[s, a[l]:a[l] + S.bonds[n][l], b[r]:b[r] + S.bonds[1 - n][r]] for s, l, r in S.mps(n)])


def dense_bm(S, b, keys, v):
    X, o = torch.zeros(S.dim[b], S.dim[b], dtype=v.dtype, device="cuda"), 0
    for p, q in keys:
        r, c = S.bonds[b][p], S.bonds[b][q]
        X[S.start[b][p]:S.start[b][p] + r, S.start[b][q]:S.start[b][q] + c] = v[o:o + r * c].reshape(c, r).T
        o += r * c
    return X


def flat_bm(S, b, keys, X):
    at, m = S.start[b], S.bonds[b]
    return flat([X[at[p]:at[p] + m[p], at[q]:at[q] + m[q]] for p, q in keys])


def diagonal(S, b):
    return [(q, q) for q in sorted(S.bonds[b])]


def sandwich(S, x, into):
    """v -> EHL v + v EHR + sum h (A_L part) v (A_R part), dense; `into`: flat result's layout."""
    d = S.d

    def reduced(A, side):
        out = {}
        for r, c, h in S.hnnz:
            (i0, i1), (j0, j1) = divmod(int(r), d), divmod(int(c), d)
            key, t = ((i1, j1), h * A[i0].T @ A[j0]) if side == "l" else ((i0, j0), h * A[j1] @ A[i1].T)
            out[key] = out[key] + t if key in out else t
        return out
    if into == "hac":
        L, R = reduced(dense_mps(S, 1, x["AL"]), "l"), reduced(dense_mps(S, 1, x["AR"]), "r")
        EL, ER = dense_bm(S, 0, diagonal(S, 0), x["EHL"]), dense_bm(S, 1, diagonal(S, 1), x["EHR"])

        def f(V):
            out = EL @ V + V @ ER
            for (i, j), M in L.items():
                out[i] += M @ V[j]
            for (i, j), M in R.items():
                out[i] += V[j] @ M
            return out
        return f
    AL, AR = dense_mps(S, 1, x["AL"]), dense_mps(S, 0, x["AR"])
    EL, ER = (dense_bm(S, 0, diagonal(S, 0), x[k]) for k in ("EHL", "EHR"))
    L = reduced(AL, "l")

    def g(V):
        out = EL @ V + V @ ER
        for (i, j), M in L.items():
            out += M @ V @ AR[j] @ AR[i].T
        return out
    return g


def transfer(S, case, lower, upper):
    order = (0, 1) if case["dir"] == "l" else (1, 0)

    def f(X):
        for n in order:
            A, U = lower[n].to(X.dtype), upper[n].to(X.dtype)
            if case["dir"] == "l":
                X = sum(U[s].T @ (X @ A[s]) for s in range(S.d))
            else:
                X = sum((A[s] @ X) @ U[s].T for s in range(S.d))
        return X
    return f


def neumann(step, b, most=4000):
    """The sum of step^k b: (1 - step)^-1 b for a contraction."""
    y, t, scale = b.clone(), b, torch.linalg.norm(b).item()
    for k in range(most):
        t = step(t)
        y += t
        if k % 16 == 15 and torch.linalg.norm(t).item() < 1e-17 * scale:
            return y
    return None


def exact(case, seed):
    op = case["op"]
    S, x = inputs(case, seed)
    if op == "hac":
        return flat_mps(S, 0, sandwich(S, x, "hac")(dense_mps(S, 0, x["v"])))
    if op == "hc":
        k = diagonal(S, 0)
        return flat_bm(S, 0, k, sandwich(S, x, "hc")(dense_bm(S, 0, k, x["v"])))
    if op in ("tm", "tmproj", "env"):
        k = diagonal(S, 0)
        A = [dense_mps(S, n, x["A%d" % n]) for n in (0, 1)]
        T = transfer(S, case, A, A)
        X, rho, one = (dense_bm(S, 0, k, v) for v in (x["v"], x["rho"], eye(S, 0)))
        if op == "tm":
            return flat_bm(S, 0, k, T(X))
        proj = lambda Y: torch.sum(Y * rho.T) * one
        if op == "tmproj":
            return flat_bm(S, 0, k, X - T(X) + proj(X))
        # 1 is T's fixed point and proj(1) = 1: T - proj is the contraction, and T proj = proj
        y = neumann(lambda Y: T(Y) - proj(Y), X - proj(X))
        return None if y is None else flat_bm(S, 0, k, y)
    if op == "lanczos":
        return exact_lanczos(S, x)
    if op == "qr":
        M = split_mps(S, 0, x["v"])
        Q, R = {}, []
        for q in sorted(S.bonds[1]):
            keys = [k for k in M if M[k][0] == q]
            if not keys:
                continue
            Y, T = torch.linalg.qr(torch.cat([M[k][1] for k in keys]))
            sign = torch.where(T.diagonal() < 0, -1.0, 1.0).to(F64)
            Y, o = Y * sign, 0
            R.append(T * sign[:, None])
            for k in keys:
                Q[k] = Y[o:o + M[k][1].shape[0]]
                o += M[k][1].shape[0]
        P, R2, o = [], [], 0
        for q, m in sorted(S.bonds[1].items()):
            Y, T = torch.linalg.qr(x["c"][o:o + m * m].reshape(m, m).T)
            sign = torch.where(T.diagonal() < 0, -1.0, 1.0).to(F64)
            P.append(Y * sign)
            R2.append(T * sign[:, None])
            o += m * m
        return [flat([Q[(s, l)] for s, l, _ in S.mps(0)]), flat(R), flat(P), flat(R2)]
    if op == "polar":
        out, values = [], []
        for side in "lr":
            M = split_mps(S, 0, x[side])
            sv, W = [], {}
            for q in sorted(S.bonds[1] if side == "l" else S.bonds[0]):
                keys = [k for k in M if (M[k][0] if side == "l" else k[1]) == q]
                if not keys:
                    continue
                U, s, V = torch.linalg.svd(torch.cat([M[k][1] for k in keys], 0 if side == "l" else 1).cpu(),
                                           full_matrices=False)
                sv.append(s)
                P, o = (U @ V).cuda(), 0
                for k in keys:
                    w = M[k][1].shape[0 if side == "l" else 1]
                    W[k] = P[o:o + w] if side == "l" else P[:, o:o + w]
                    o += w
            out.append(flat([W[(s, l)] for s, l, _ in S.mps(0)]))
            values.append(torch.cat(sv))
        return out + values
    keys = S.mixed(0)
    T = transfer(S, case, [dense_mps(S, n, x["A%d" % n]) for n in (0, 1)],
                 [dense_mps(S, n, x["B%d" % n]) for n in (0, 1)])
    # a real operator on a complex matrix: real and imaginary parts by themselves
    both = lambda Y: torch.complex(T(Y.real.contiguous()), T(Y.imag.contiguous()))
    fac = complex(math.cos(x["p"]), math.sin(x["p"]))
    y = neumann(lambda Y: fac * both(Y), dense_bm(S, 0, keys, torch.complex(x["re"], x["im"])))
    if y is None:
        return [None, None]
    return [flat_bm(S, 0, keys, y.real), flat_bm(S, 0, keys, y.imag)]


def exact_lanczos(S, x, steps=320):
    """The lowest eigenpair of H_AC by an unrestarted, fully reorthogonalised Lanczos run."""
    f = sandwich(S, x, "hac")
    n = S.mps_size(0)
    steps = min(steps, n - 1)
    V = torch.zeros(steps + 1, n, dtype=F64, device="cuda")
    V[0] = x["v"] / torch.linalg.norm(x["v"])
    T = np.zeros((steps + 1, steps + 1))
    for k in range(steps):
        w = flat_mps(S, 0, f(dense_mps(S, 0, V[k])))
        for _ in range(2):
            h = V[:k + 1] @ w
            T[k, k] += h[k].item()
            w = w - h @ V[:k + 1]
        b = torch.linalg.norm(w).item()
        V[k + 1] = w / b
        T[k, k + 1] = T[k + 1, k] = b
        if k % 16 == 15 or k == steps - 1:
            e, y = np.linalg.eigh(T[:k + 1, :k + 1])
            if abs(b * y[-1, 0]) < 1e-15 * abs(e[0]):
                v = torch.from_numpy(y[:, 0]).cuda() @ V[:k + 1]
                return {"energy": float(e[0]), "vector": v * torch.sign(torch.dot(v, x["v"]))}
    return None
