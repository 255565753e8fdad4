"""The operator applies of this framework as a user's program calls them, each
with its inputs, one pass and its result in plain 64-bit torch.

The applies are called through the package's public entry points with device
tensors that the program keeps: bk1_apply (mass), bk3_apply (Poisson, with and
without a coefficient), bk5_apply (collocated Laplacian, with and without the
mass term), bk3_adjoint (the gradient with respect to the coefficient and the
geometric factors) and the mixed-order Helmholtz plan's apply and CG solve.
Geometry: every element is a cube of edge 1 whose eight corners are moved by up
to 0.15 in each direction (a trilinear map); u ~ U[-1, 1], log k ~ N(0, 0.5^2).
"""
import math

import numpy as np
import torch

import omp_bk_gb300 as bk
from omp_bk_gb300 import helmholtz

PRECS = {"fp64": bk.PREC_FP64, "fp32": bk.PREC_FP32, "mixed": bk.PREC_MIXED}
LAYOUTS = {"factor": bk.LAYOUT_FACTOR, "interleaved": bk.LAYOUT_INTERLEAVED, "column": bk.LAYOUT_COLUMN}
# points of the six factors (f, i, j, k) in each layout's order
G_ORDER = {"factor": (0, 1, 2, 3, 4), "interleaved": (0, 2, 3, 1, 4), "column": (0, 1, 4, 2, 3)}
JITTER = 0.15


def listed():
    return [
        # a call on a handful of elements (a coarse level, a unit test): latency
        {"name": "bk1_p2_few", "op": "bk1", "p": 2, "E": 37, "prec": "fp64"},
        # the CEED mass apply at its small configuration, L2-resident
        {"name": "bk1_p3_fp64", "op": "bk1", "p": 3, "E": 4096, "prec": "fp64"},
        # a large mass apply in the reference drivers' float
        {"name": "bk1_p6_fp32", "op": "bk1", "p": 6, "E": 60013, "prec": "fp32"},
        # the Poisson apply in plain FP64 at its configuration's size
        {"name": "bk3_p6_fp64", "op": "bk3", "p": 6, "E": 131072, "prec": "fp64", "coef": False, "gform": "plain"},
        # the same operator in the mixed form of a refined solver
        {"name": "bk3_p6_mixed", "op": "bk3", "p": 6, "E": 131072, "prec": "mixed", "coef": False, "gform": "plain"},
        # a variable-coefficient forward apply at an odd size
        {"name": "bk3_p4_mixed_coef", "op": "bk3", "p": 4, "E": 20011, "prec": "mixed", "coef": True,
         "gform": "plain"},
        # the collocated Laplacian in plain FP64, 134 M points: the largest call
        {"name": "bk5_p7_fp64", "op": "bk5", "p": 7, "E": 262144, "prec": "fp64", "layout": "column", "mass": False,
         "gform": "plain"},
        # an ordinary FP64 apply on the default (interleaved) layout, odd size
        {"name": "bk5_p4_fp64_interleaved", "op": "bk5", "p": 4, "E": 9973, "prec": "fp64", "layout": "interleaved",
         "mass": False, "gform": "plain"},
        # the single-order Helmholtz operator of a mixed-precision solver
        {"name": "bk5_p3_mixed_mass", "op": "bk5", "p": 3, "E": 125003, "prec": "mixed", "layout": "column",
         "mass": True, "gform": "plain"},
        # the backward pass of the variable-coefficient operator
        {"name": "adjoint_p4_fp64", "op": "adjoint", "p": 4, "E": 65536, "prec": "fp64", "gform": "plain"},
        # the mixed-order operator, p = 2..8, 43.5 M points in one launch
        {"name": "helmholtz_mixed", "op": "helmholtz", "base": 4096, "first": 2, "last": 8, "prec": "mixed"},
        # a whole solve to 1e-10 with FP64 refinement
        {"name": "helmholtz_cg", "op": "cg", "base": 512, "first": 2, "last": 8, "prec": "mixed"},
    ]


def draw(rng):
    """One more apply: any operator, order, storage and option, from a few
    elements to tens of millions of points."""
    op = rng.choice(["bk1", "bk1", "bk3", "bk3", "bk3", "bk5", "bk5", "bk5", "adjoint", "helmholtz"])
    if op == "helmholtz":
        first = rng.randint(2, 6)
        last = rng.randint(first + 1, 8)
        base = max(1, round(math.exp(rng.uniform(math.log(2), math.log(4096)))))
        return {"op": op, "base": base, "first": first, "last": last, "prec": rng.choice(["mixed", "mixed", "fp64"])}
    p = rng.randint(1, 8)
    q = p + 1 if op == "bk5" else p + 2
    points = math.exp(rng.uniform(math.log(3e3), math.log(6e7 if op != "adjoint" else 2e7)))
    E = max(1, int(points / q ** 3)) + rng.choice([0, 1])
    prec = rng.choice(["fp64", "fp64", "mixed", "fp32"])
    case = {"op": op, "p": p, "E": E, "prec": prec}
    if op in ("bk3", "bk5", "adjoint"):
        case["gform"] = "split" if prec == "fp64" and rng.random() < 0.25 else "plain"
    if op == "bk3":
        case["coef"] = rng.random() < 0.4
    if op == "bk5":
        case["layout"] = rng.choice(["factor", "interleaved", "column", "column"])
        case["mass"] = rng.random() < 0.4
    return case


# ---- rules and matrices in numpy ---------------------------------------------------

def _gll(n):
    c = np.zeros(n)
    c[-1] = 1.0
    x = np.concatenate([[-1.0], np.sort(np.polynomial.legendre.legroots(np.polynomial.legendre.legder(c)).real), [1.0]])
    x = 0.5 * (x - x[::-1])
    w = 2.0 / (n * (n - 1) * np.polynomial.legendre.legval(x, c) ** 2)
    return x, w


def _lagrange(nodes, pts):
    """l_i(pts[p]) as [p, i]."""
    return np.array([[np.prod([(t - nodes[m]) / (nodes[i] - nodes[m]) for m in range(len(nodes)) if m != i])
                      for i in range(len(nodes))] for t in pts])


def _deriv(x):
    """l_n'(x_i) as [i, n]."""
    n = len(x)
    w = np.array([1.0 / np.prod([x[i] - x[m] for m in range(n) if m != i]) for i in range(n)])
    D = np.array([[(w[j] / w[i]) / (x[i] - x[j]) if i != j else 0.0 for j in range(n)] for i in range(n)])
    return D - np.diag(D.sum(axis=1))


def _rules(op, p):
    """(points, weights, interpolation [point, node] or None, derivative [point, point])."""
    if op in ("bk1", "bk3", "adjoint"):
        x, w = np.polynomial.legendre.leggauss(p + 2)
        return x, w, _lagrange(_gll(p + 1)[0], x), _deriv(x)
    x, w = _gll(p + 1)
    return x, w, None, _deriv(x)


# ---- inputs ------------------------------------------------------------------------

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _uniform(gen, n, dtype=torch.float64):
    return torch.rand(n, generator=gen, device="cuda", dtype=torch.float64).mul_(2).sub_(1).to(dtype)


def _geometry(gen, E, x, w, layout=None, want_mass=False, dtype=torch.float64):
    """G (w detJ J^-1 J^-T, six factors, in `layout`) and w detJ of E jittered
    unit cubes at the tensor points x."""
    Q = len(x)
    t = torch.tensor(x, device="cuda", dtype=torch.float64)
    wt = torch.tensor(w, device="cuda", dtype=torch.float64)
    w3 = (wt[:, None, None] * wt[None, :, None] * wt[None, None, :])
    n, d = torch.stack([(1 - t) / 2, (1 + t) / 2]), torch.stack([torch.full_like(t, -0.5), torch.full_like(t, 0.5)])
    # derivative of corner (a, b, c)'s shape function along each direction
    dN = torch.stack([torch.einsum("ai,bj,ck->abcijk", *[d if r == s else n for s in range(3)]) for r in range(3)])
    dN = dN.reshape(3, 8, Q ** 3).permute(1, 0, 2).reshape(8, 3 * Q ** 3)
    cube = torch.tensor([[a, b, c] for a in (0, 1) for b in (0, 1) for c in (0, 1)], device="cuda",
                        dtype=torch.float64)
    G = torch.empty(E * 6 * Q ** 3, device="cuda", dtype=dtype) if layout is not None else None
    M = torch.empty(E * Q ** 3, device="cuda", dtype=dtype) if want_mass else None
    step = max(1, (1 << 24) // Q ** 3)
    for e0 in range(0, E, step):
        ne = min(step, E - e0)
        corners = cube + JITTER * (torch.rand(ne, 8, 3, generator=gen, device="cuda", dtype=torch.float64) * 2 - 1)
        # J[:, a, r] = d x_a / d xi_r
        J = (corners.transpose(1, 2).reshape(ne * 3, 8) @ dN).reshape(ne, 3, 3, Q, Q, Q)
        c = [[J[:, (a + 1) % 3, (r + 1) % 3] * J[:, (a + 2) % 3, (r + 2) % 3]
              - J[:, (a + 1) % 3, (r + 2) % 3] * J[:, (a + 2) % 3, (r + 1) % 3] for r in range(3)] for a in range(3)]
        det = sum(J[:, a, 0] * c[a][0] for a in range(3))
        if M is not None:
            M[e0 * Q ** 3:(e0 + ne) * Q ** 3] = (w3 * det).reshape(-1).to(dtype)
        if G is not None:
            s = w3 / det
            g = torch.stack([s * sum(c[a][r] * c[a][u] for a in range(3))
                             for r, u in ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))], dim=1)
            g = g.permute(*G_ORDER[layout]).reshape(-1)
            G[e0 * 6 * Q ** 3:(e0 + ne) * 6 * Q ** 3] = g.to(dtype)
    return G, M


def _orders(case):
    return [(p, case["base"] * 2 ** (case["last"] - p)) for p in range(case["first"], case["last"] + 1)]


def _mixed_inputs(case, seed):
    """u, G (column layout) and mass of every order one after another, in FP64."""
    gen = _generator(seed)
    G, M = [], []
    for p, E in _orders(case):
        x, w = _gll(p + 1)
        g, m = _geometry(gen, E, x, w, "column", True)
        G.append(g)
        M.append(m)
    n = sum(m.numel() for m in M)
    return _uniform(gen, n), torch.cat(G), torch.cat(M)


def _inputs(case, seed):
    """The tensors of a single-order case in its storage type."""
    op, p, E = case["op"], case["p"], case["E"]
    dt = torch.float64 if case["prec"] == "fp64" else torch.float32
    x, w, _, _ = _rules(op, p)
    Q, P = len(x), p + 1
    gen = _generator(seed)
    t = {"u": _uniform(gen, E * P ** 3, dt)}
    if op == "bk1":
        t["q"] = _geometry(gen, E, x, w, None, True, dt)[1]
        return t
    layout = case.get("layout", "factor")
    t["G"], m = _geometry(gen, E, x, w, layout, bool(case.get("mass")), dt)
    if m is not None:
        t["mass"] = m
    if case.get("coef") or op == "adjoint":
        t["k"] = torch.exp(0.5 * torch.randn(E * Q ** 3, generator=gen, device="cuda", dtype=torch.float64)).to(dt)
    if op == "adjoint":
        t["res"] = _uniform(gen, E * P ** 3, dt)
    return t


def prepare(case, seed):
    op = case["op"]
    s = {"op": op, "prec": PRECS[case["prec"]]}
    if op in ("helmholtz", "cg"):
        u, G, M = _mixed_inputs(case, seed)
        s["plan"] = helmholtz.HelmholtzPlan(_orders(case))
        if op == "cg":
            s.update(G64=G, M64=M, G32=G.float(), M32=M.float(), x=torch.empty_like(u), f=_helmholtz(case, u, G, M))
        else:
            dt = torch.float64 if case["prec"] == "fp64" else torch.float32
            s.update(G=G.to(dt), mass=M.to(dt), u=u.to(dt))
            s["v"] = torch.empty_like(s["u"])
        return s
    p = case["p"]
    s.update(_inputs(case, seed), p=p, E=case["E"])
    s["gform"] = bk.G_FF if case.get("gform") == "split" else bk.G_STORAGE
    if s["gform"] == bk.G_FF:
        s["G"] = bk.g_to_ff(s["G"])
    if op == "bk5":
        s["D"] = bk.bk5_matrices(p)[0]
        s["layout"] = LAYOUTS[case["layout"]]
    else:
        s["B"], s["D"] = bk.bk1_bk3_matrices(p)[:2]
    if op == "adjoint":
        s["dk"], s["dG"] = torch.empty_like(s["k"]), torch.empty_like(s["G"])
    else:
        s["v"] = torch.empty_like(s["u"])
    return s


def run(s):
    op = s["op"]
    if op == "bk1":
        bk.bk1_apply(s["p"], s["E"], s["B"], s["q"], s["u"], s["v"], prec=s["prec"])
        return s["v"]
    if op == "bk3":
        bk.bk3_apply(s["p"], s["E"], s["B"], s["D"], s["G"], s["u"], s["v"], k=s.get("k"), prec=s["prec"],
                     gform=s["gform"])
        return s["v"]
    if op == "bk5":
        bk.bk5_apply(s["p"], s["E"], s["D"], s["G"], s["u"], s["v"], prec=s["prec"], layout=s["layout"],
                     mass=s.get("mass"), lam=1.0, gform=s["gform"])
        return s["v"]
    if op == "adjoint":
        bk.bk3_adjoint(s["p"], s["E"], s["B"], s["D"], s["G"], s["k"], s["u"], s["res"], s["dk"], s["dG"],
                       prec=s["prec"], gform=s["gform"])
        return [s["dk"], s["dG"]]
    if op == "helmholtz":
        s["plan"].apply(s["G"], s["mass"], 1.0, s["u"], s["v"], prec=s["prec"])
        return s["v"]
    s["x"].zero_()
    s["plan"].cg(s["G64"], s["M64"], s["G32"], s["M32"], 1.0, s["f"], s["x"])
    return s["x"]


# ---- what a pass cannot do without ---------------------------------------------------

def work(case):
    """Bytes: inputs once, outputs once.  Flops: the sum-factorised
    contractions in their even-odd form (a line of m values into n takes m n
    flops) and the products at the points."""
    op = case["op"]
    size = 8 if case["prec"] == "fp64" else 4
    if op in ("helmholtz", "cg"):
        points = sum(E * (p + 1) ** 3 for p, E in _orders(case))
        flops = sum(E * (p + 1) ** 3 * (6 * (p + 1) + 20) for p, E in _orders(case))
        if op == "cg":   # both forms of the operator, f and x once; one apply
            return {"bytes": points * (7 * 12 + 16), "flops": flops}
        return {"bytes": points * size * 9, "flops": flops}
    p, E = case["p"], case["E"]
    P, Q = p + 1, (p + 1 if op == "bk5" else p + 2)
    q3 = E * Q ** 3
    there = E * (P ** 3 * Q + P ** 2 * Q ** 2 + P * Q ** 3)   # nodes to points
    if op == "bk1":
        return {"bytes": size * (2 * E * P ** 3 + q3), "flops": 2 * there + q3}
    if op == "bk3":
        k = 1 if case["coef"] else 0
        return {"bytes": size * (2 * E * P ** 3 + (6 + k) * q3), "flops": 2 * there + q3 * (6 * Q + 17 + 3 * k)}
    if op == "bk5":
        k = 1 if case["mass"] else 0
        return {"bytes": size * (2 * E * P ** 3 + (6 + k) * q3), "flops": q3 * (6 * Q + 17 + 3 * k)}
    return {"bytes": size * (2 * E * P ** 3 + 14 * q3), "flops": 2 * there + q3 * (6 * Q + 40)}


# ---- the results in plain 64-bit torch ---------------------------------------------

def _along(M, x):
    """M ([out, in]) along each of the three point directions of x (E, i, j, k)."""
    for d in (1, 2, 3):
        x = torch.movedim(torch.tensordot(x, M, dims=([d], [1])), -1, d)
    return x


def _one(M, x, d):
    return torch.movedim(torch.tensordot(x, M, dims=([d], [1])), -1, d)


def _fluxes(g, q):
    """The fluxes of gradient q (three (E, i, j, k)) with factors g (E, 6, i, j, k)."""
    return [g[:, 0] * q[0] + g[:, 1] * q[1] + g[:, 2] * q[2],
            g[:, 1] * q[0] + g[:, 3] * q[1] + g[:, 4] * q[2],
            g[:, 2] * q[0] + g[:, 4] * q[1] + g[:, 5] * q[2]]


def _factors(G, E, Q, layout):
    """G (E, 6, i, j, k) in 64 bits from its stored layout."""
    order = G_ORDER[layout]
    shape = [(E, 6, Q, Q, Q)[a] for a in order]
    back = [order.index(a) for a in range(5)]
    return G.reshape(shape).permute(*back).double()


def _laplacian(D, g, u):
    f = _fluxes(g, [_one(D, u, d) for d in (1, 2, 3)])
    return sum(_one(D.T, f[d - 1], d) for d in (1, 2, 3))


def _device(a):
    return torch.tensor(a, device="cuda", dtype=torch.float64)


def _helmholtz(case, u, G, M):
    """(K + M) u of the mixed orders, in 64 bits."""
    out = torch.empty(u.numel(), device="cuda", dtype=torch.float64)
    o = 0
    for p, E in _orders(case):
        Q = p + 1
        D = _device(_deriv(_gll(Q)[0]))
        n = E * Q ** 3
        w = u[o:o + n].double().reshape(E, Q, Q, Q)
        g = _factors(G[6 * o:6 * (o + n)], E, Q, "column")
        out[o:o + n] = (_laplacian(D, g, w) + M[o:o + n].double().reshape(w.shape) * w).reshape(-1)
        o += n
    return out


def exact(case, seed):
    op = case["op"]
    if op in ("helmholtz", "cg"):
        u, G, M = _mixed_inputs(case, seed)
        if op == "cg":
            return u   # f was made from it
        dt = torch.float64 if case["prec"] == "fp64" else torch.float32
        return _helmholtz(case, u.to(dt), G.to(dt), M.to(dt))
    t = _inputs(case, seed)
    p, E = case["p"], case["E"]
    _, _, B, D = _rules(op, p)
    D, P, Q = _device(D), p + 1, len(D)
    u = t["u"].double().reshape(E, P, P, P)
    if op == "bk5":
        v = _laplacian(D, _factors(t["G"], E, Q, case["layout"]), u)
        if "mass" in t:
            v = v + t["mass"].double().reshape(u.shape) * u
        return v.reshape(-1)
    B = _device(B)
    if op == "bk1":
        return _along(B.T, _along(B, u) * t["q"].double().reshape(E, Q, Q, Q)).reshape(-1)
    g = _factors(t["G"], E, Q, "factor")
    if op == "bk3":
        if "k" in t:
            g = g * t["k"].double().reshape(E, 1, Q, Q, Q)
        return _along(B.T, _laplacian(D, g, _along(B, u))).reshape(-1)
    k = t["k"].double().reshape(E, Q, Q, Q)
    wu, wr = _along(B, u), _along(B, t["res"].double().reshape(E, P, P, P))
    qu, qr = [_one(D, wu, d) for d in (1, 2, 3)], [_one(D, wr, d) for d in (1, 2, 3)]
    f = _fluxes(g, qu)
    dk = sum(a * b for a, b in zip(qr, f))
    pairs = ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))
    dG = torch.stack([k * (qr[a] * qu[b] + (qr[b] * qu[a] if a != b else 0)) for a, b in pairs], dim=1)
    return [dk.reshape(-1), dG.reshape(-1)]
