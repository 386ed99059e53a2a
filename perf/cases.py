"""The work whose speed is measured: element operators of hexahedra, prisms and
tetrahedra, a mixed mesh's collections in one batched call, and the conjugate
gradient solve that is built on them.

Three kinds of case:

* "op": one collection operator applied to device buffers, as a solver's time
  step does. `nq` is the number of points in the first direction: nm + 1, or more
  where a nonlinear term is over-integrated. `curved` elements carry geometric
  factors at every point, straight-sided ones a single set.
* "batch": every collection of a mixed mesh (three shapes, several orders)
  applied in one call.
* "solve": a Helmholtz solve on a curved box of n^3 hexahedra, from a local
  right-hand side to the local solution.
"""
import math

import numpy as np
import torch

import nektar_b200 as nb

SHAPES = ("hex", "prism", "tet")
OPS = ("helmholtz", "linear_adr", "bwdtrans", "iproduct", "iproduct_deriv", "physderiv")
# geometric values an operator needs per point of a curved element (per straight-sided
# element): the Jacobian and six metric terms, nine derivative factors, the Jacobian
GEOMETRY = {"helmholtz": 7, "linear_adr": 7, "bwdtrans": 0, "iproduct": 1,
            "iproduct_deriv": 9, "physderiv": 9}
LISTED_BYTES = 1.2e9  # about the largest listed pass of an operator
AMP = 0.05            # curvature of the solve's box


def op_case(name, op, shape, nm, elements, nq=None, precision="fp64", curved=True):
    c = {"kind": "op", "op": op, "shape": shape, "nm": nm, "nq": nq or nm + 1,
         "elements": elements, "precision": precision, "curved": curved}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a coarse mesh, or one rank's share of a strongly scaled one: latency counts
        op_case("hex_helmholtz_small", "helmholtz", "hex", 4, 64),
        # the matrix-vector product of the largest solve
        op_case("hex_helmholtz_large", "helmholtz", "hex", 7, 32 ** 3),
        # the same at a higher order in the mixed-precision solve's inner iterations
        op_case("hex_helmholtz_fp32", "helmholtz", "hex", 9, 24 ** 3, precision="fp32"),
        # boundary-layer prisms of a straight-sided mesh
        op_case("prism_helmholtz_straight", "helmholtz", "prism", 6, 2 * 18 ** 3, curved=False),
        # a curved tetrahedral mesh
        op_case("tet_helmholtz_curved", "helmholtz", "tet", 7, 6 * 12 ** 3),
        # an implicit advection-diffusion step; an element count that fills nothing evenly
        op_case("hex_adr_odd_order", "linear_adr", "hex", 8, 9259),
        # to physical space at the start of a step
        op_case("prism_bwdtrans", "bwdtrans", "prism", 5, 2 * 19 ** 3),
        # from an over-integrated nonlinear term back to coefficients
        op_case("hex_iproduct_overint", "iproduct", "hex", 4, 22 ** 3, nq=8),
        # gradients of the velocity for the nonlinear term
        op_case("hex_physderiv", "physderiv", "hex", 7, 24 ** 3),
        # a weak divergence on straight-sided tetrahedra
        op_case("tet_iproduct_deriv_straight", "iproduct_deriv", "tet", 5, 6 * 16 ** 3,
                curved=False),
        # a mixed mesh of variable order in one call
        {"name": "mixed_mesh_batch", "kind": "batch", "op": "helmholtz", "cells": 9000,
         "nm_low": 3, "nm_high": 8, "precision": "fp64", "curved": True},
        # the implicit solve of a time step
        {"name": "hex_solve", "kind": "solve", "n": 14, "nm": 7, "mixed": False},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choices(("op", "batch", "solve"), (10, 1, 1))[0]
    while True:
        if kind == "op":
            op, shape = rng.choice(OPS), rng.choice(SHAPES)
            nm = rng.randint(3, 10)
            nq = nm + 1 if rng.random() < 0.8 else rng.randint(nm + 2, min(2 * nm, 12))
            c = op_case(None, op, shape, nm, 1, nq, rng.choice(("fp64", "fp64", "fp32")),
                        rng.random() < 0.6)
            most = int(LISTED_BYTES / _op_bytes(c))
            c["elements"] = _log_int(rng, 40, min(most, 60000))
        elif kind == "batch":
            low = rng.randint(3, 5)
            c = {"kind": "batch", "op": rng.choice(OPS), "cells": _log_int(rng, 100, 9000),
                 "nm_low": low, "nm_high": rng.randint(low + 1, 8),
                 "precision": rng.choice(("fp64", "fp32")), "curved": rng.random() < 0.7}
        else:
            c = {"kind": "solve", "n": rng.randint(4, 14), "nm": rng.randint(3, 7),
                 "mixed": rng.random() < 0.5}
        if kind == "solve" or work(c)["bytes"] <= LISTED_BYTES:
            return c


# ---- sizes -------------------------------------------------------------------


def _points_per_direction(shape, nq):
    return {"hex": (nq, nq, nq), "prism": (nq, nq, nq - 1), "tet": (nq, nq - 1, nq - 1)}[shape]


def _nt(shape, nq):
    return math.prod(_points_per_direction(shape, nq))


def _in_out(op, nc, nt):
    """(input, output) values per element."""
    return {"helmholtz": (nc, nc), "linear_adr": (nc, nc), "bwdtrans": (nc, nt),
            "iproduct": (nt, nc), "iproduct_deriv": (3 * nt, nc), "physderiv": (nt, 3 * nt)}[op]


def _op_bytes(c):
    nc, nt = nb.ncoeffs(c["shape"], c["nm"]), _nt(c["shape"], c["nq"])
    vals = sum(_in_out(c["op"], nc, nt))
    if c["op"] == "linear_adr":
        vals += 3 * nt  # advection varies from point to point on any mesh
    vals += GEOMETRY[c["op"]] * (nt if c["curved"] else 1)
    return c["elements"] * vals * (8 if c["precision"] == "fp64" else 4)


def _op_flops(c):
    nm, (q0, q1, q2) = c["nm"], _points_per_direction(c["shape"], c["nq"])
    nc, nt = nb.ncoeffs(c["shape"], nm), q0 * q1 * q2
    # one pass between coefficients and points, one gradient
    if c["shape"] == "hex":
        trans = 2 * (q0 * nm ** 3 + q0 * q1 * nm ** 2 + nt * nm)
    elif c["shape"] == "prism":
        trans = 2 * (q2 * nc + q2 * q1 * nm ** 2 + nt * nm)
    else:
        trans = 2 * (q2 * nc + q2 * q1 * nm * (nm + 1) // 2 + nt * nm)
    grad = 2 * nt * (q0 + q1 + q2)
    per = {"helmholtz": 2 * trans + 2 * grad + 18 * nt, "linear_adr": 2 * trans + 2 * grad + 24 * nt,
           "bwdtrans": trans, "iproduct": trans + nt, "iproduct_deriv": trans + grad + 15 * nt,
           "physderiv": grad + 15 * nt}[c["op"]]
    return c["elements"] * per


def _collections(c):
    """The mixed mesh's collections, as "op" cases: a cell is one hexahedron, two
    prisms or six tetrahedra; orders are spread evenly, with a remainder."""
    orders = range(c["nm_low"], c["nm_high"] + 1)
    out = []
    for shape, share, per in zip(SHAPES, (4, 3, 2), (1, 2, 6)):
        for k, nm in enumerate(orders):
            cells = c["cells"] * share // (9 * len(orders)) + 3 * k + 1
            out.append(op_case(None, c["op"], shape, nm, cells * per, None, c["precision"],
                               c["curved"]))
    return out


def _iterations(c):
    """About the conjugate gradient iterations of a random right-hand side."""
    return 1700 * ((c["nm"] - 1) / 6) ** 1.8


def work(c):
    if c["kind"] == "op":
        return {"bytes": _op_bytes(c), "flops": _op_flops(c)}
    if c["kind"] == "batch":
        parts = [work(p) for p in _collections(c)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    p = op_case(None, "helmholtz", "hex", c["nm"], c["n"] ** 3,
                precision="fp32" if c["mixed"] else "fp64")
    size = 4 if c["mixed"] else 8
    nglob = (c["n"] * (c["nm"] - 1) + 1) ** 3
    # geometry, the map, and eleven passes over the recurrence's vectors
    nloc = c["n"] ** 3 * c["nm"] ** 3
    per = 7 * _nt("hex", c["nm"] + 1) * c["n"] ** 3 * size
    per += 4 * nloc + 11 * nglob * size
    it = _iterations(c)
    return {"bytes": it * per, "flops": it * (_op_flops(p) + 12 * nglob)}


def tolerance(c):
    # about four times the largest distance from exact() that was seen over the
    # ranges: the orders of magnitude of rounding over a few hundred terms, and of a
    # solution whose residual is 1e-10 of the right-hand side
    if c["kind"] == "solve":
        return {"rel": 2e-10}
    if c["precision"] == "fp32":
        return {"rel": 4e-6}
    return {"rel": 2e-14}


# ---- what a program has before the call -----------------------------------------


def _uniform(gen, *shape):
    return torch.rand(*shape, generator=gen, dtype=torch.float64, device="cuda") * 2 - 1


def _geometry(c, gen):
    """jac and df[k*3+j] = d xi_j / d x_k of small sheared, stretched and (curved)
    point-wise varying elements, in the Collections layout."""
    E = c["elements"]
    n = E * _nt(c["shape"], c["nq"]) if c["curved"] else E
    h = max(2.0, E ** (1 / 3))
    jac = (1 + 0.3 * _uniform(gen, n)) / (2 * h) ** 3
    df = 0.25 * _uniform(gen, 9, n)
    df[0] += 1
    df[4] += 1
    df[8] += 1
    return jac, (2 * h * df).contiguous()


def _inputs(c, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    jac, df = _geometry(c, gen)
    nc, nt = nb.ncoeffs(c["shape"], c["nm"]), _nt(c["shape"], c["nq"])
    dtype = torch.float64 if c["precision"] == "fp64" else torch.float32
    x = _uniform(gen, c["elements"] * _in_out(c["op"], nc, nt)[0]).to(dtype)
    lam = 1.0 + 0.5 * float(_uniform(gen, 1)[0])
    vel = _uniform(gen, 3, c["elements"] * nt) if c["op"] == "linear_adr" else None
    return jac, df, x, lam, vel


def _operator(c, jac, df, lam, vel):
    T, nq = nb.shape_tables(c["shape"], c["nm"], c["nq"])
    op = nb.Operator(c["op"], shape=c["shape"], nm=c["nm"], nq=nq, nelmt=c["elements"], T=T,
                     jac=jac, df=df, deformed=c["curved"], precision=c["precision"])
    if c["op"] in ("helmholtz", "linear_adr"):
        op.set_factors(lam)
    if vel is not None:
        op.set_varcoeffs(*[v.data_ptr() for v in vel])
    return op


def _solve_inputs(c, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    lam = 1.0 + 0.5 * float(_uniform(gen, 1)[0])
    return _uniform(gen, c["n"] ** 3 * c["nm"] ** 3) / c["n"] ** 3, lam


def prepare(case, seed):
    c = case
    if c["kind"] == "op":
        jac, df, x, lam, vel = _inputs(c, seed)
        op = _operator(c, jac, df, lam, vel)
        outs = [torch.empty(op.out_size, dtype=x.dtype, device="cuda")
                for _ in range(3 if c["op"] == "physderiv" else 1)]
        return {"kind": "op", "op": op, "x": x, "outs": outs}
    if c["kind"] == "batch":
        ops, xs = [], []
        for k, p in enumerate(_collections(c)):
            jac, df, x, lam, vel = _inputs(p, 1000 * seed + k)
            ops.append(_operator(p, jac, df, lam, vel))
            xs.append(x)
        batch = nb.Batch(ops)
        x = torch.cat(xs)
        return {"kind": "batch", "op": batch, "x": x,
                "out": torch.empty(batch.out_size, dtype=x.dtype, device="cuda")}
    b, lam = _solve_inputs(c, seed)
    mesh = nb.BoxMesh("hex", c["n"], c["nm"], c["nm"] + 1, amp=AMP, geom_device=0)
    ops = [nb.Operator("helmholtz", mesh)]
    ops32 = [nb.Operator("helmholtz", mesh, precision="fp32")] if c["mixed"] else None
    for op in ops + (ops32 or []):
        op.set_factors(lam)
    system = nb.GlobalLinSys(ops, *mesh.assembly(), ops32=ops32)
    return {"kind": "solve", "op": system, "mixed": c["mixed"], "b": b, "x": torch.empty_like(b)}


def run(state):
    op, stream = state["op"], torch.cuda.current_stream().cuda_stream
    if state["kind"] == "op":
        op.apply_device(state["x"].data_ptr(), *[o.data_ptr() for o in state["outs"]],
                        stream=stream)
        return state["outs"]
    if state["kind"] == "batch":
        op.apply_device(state["x"].data_ptr(), state["out"].data_ptr(), stream=stream)
        return state["out"]
    x = state["x"].zero_()  # homogeneous Dirichlet values
    op.solve_device(state["b"].data_ptr(), x.data_ptr(), tol=1e-10, stream=stream,
                    mixed=state["mixed"])
    return x


# ---- the same in 64 bits, from the definitions ---------------------------------------


def _jacobi(n, a, b, z):
    """P_n^{a,b} at z."""
    p0, p1 = np.ones_like(z), 0.5 * (a - b + (a + b + 2) * z)
    if n == 0:
        return p0
    for k in range(2, n + 1):
        s = 2 * k + a + b
        p0, p1 = p1, (((s - 1) * (a * a - b * b + s * (s - 2) * z) * p1
                       - 2 * (k + a - 1) * (k + b - 1) * s * p0)
                      / (2 * k * (k + a + b) * (s - 2)))
    return p1


def _jacobi_zeros(n, a, b):
    """Zeros of P_n^{a,b}: eigenvalues of the recurrence's matrix, then Newton."""
    if n == 0:
        return np.zeros(0)
    k = np.arange(n)
    s = 2 * k + a + b
    diag = np.array([(b * b - a * a) / (t * (t + 2)) if t * (t + 2) else (b - a) / (a + b + 2)
                     for t in s])
    k, s = k[1:], s[1:]
    off = np.sqrt(4 * k * (k + a) * (k + b) * (k + a + b) / (s * s * (s + 1) * (s - 1)))
    z = np.linalg.eigvalsh(np.diag(diag) + np.diag(off, 1) + np.diag(off, -1))
    for _ in range(3):
        z = z - _jacobi(n, a, b, z) / (0.5 * (n + a + b + 1) * _jacobi(n - 1, a + 1, b + 1, z))
    return z


def _rule(alpha, n):
    """Points, weights and derivative matrix D[i, j] = l_j'(z_i): Gauss-Lobatto
    (alpha 0), or Gauss-Radau with the weight ((1 - z) / 2)^alpha."""
    if alpha == 0:
        z = np.concatenate(([-1.0], _jacobi_zeros(n - 2, 1, 1), [1.0]))
    else:
        z = np.concatenate(([-1.0], _jacobi_zeros(n - 1, alpha, 1)))
    diff = z[:, None] - z[None, :] + np.eye(n)
    c = diff.prod(axis=1)
    D = (c[:, None] / c[None, :]) / diff
    np.fill_diagonal(D, 0)
    np.fill_diagonal(D, -D.sum(axis=1))
    zg, wg = np.polynomial.legendre.leggauss(n + 4)
    w = np.zeros(n)
    for i in range(n):
        others = np.delete(z, i)
        li = np.prod((zg[:, None] - others) / (z[i] - others), axis=1)
        w[i] = np.sum(wg * li * ((1 - zg) / 2) ** alpha)
    return z, w, D


def _mode(p, q, z):
    """The modified basis of a collapsed direction; row p = 0 is the one of a
    Cartesian direction."""
    lo, hi = (1 - z) / 2, (1 + z) / 2
    if p == 0:
        return lo if q == 0 else hi if q == 1 else lo * hi * _jacobi(q - 2, 1, 1, z)
    a = lo ** p
    return a if q == 0 else a * hi * _jacobi(q - 1, 2 * p - 1, 1, z)


def _element(shape, nm, nq):
    """Basis (nc, nt) at the points, weights (nt), the three directions' D, and the
    factors C[a][j] of d/d xi_j = sum_a C[a][j] d/d eta_a at the points."""
    alphas = {"hex": (0, 0, 0), "prism": (0, 0, 1), "tet": (0, 1, 2)}[shape]
    rules = [_rule(a, n) for a, n in zip(alphas, _points_per_direction(shape, nq))]
    z0, z1, z2 = (r[0] for r in rules)

    def tensor(f0, f1, f2):  # first direction fastest
        return (f2[:, None, None] * f1[None, :, None] * f0[None, None, :]).ravel()

    A = [_mode(0, p, z0) for p in range(nm)]
    one0 = np.ones_like(z0)
    rows = []
    if shape == "hex":
        for r in range(nm):
            for q in range(nm):
                rows += [tensor(A[p], _mode(0, q, z1), _mode(0, r, z2)) for p in range(nm)]
    elif shape == "prism":
        for p in range(nm):
            for q in range(nm):
                for r in range(nm - p):
                    # the collapsed edge's mode does not vary along the first direction
                    f0 = one0 if (p, r) == (0, 1) else A[p]
                    rows.append(tensor(f0, _mode(0, q, z1), _mode(p, r, z2)))
    else:
        for p in range(nm):
            for q in range(nm - p):
                for r in range(nm - p - q):
                    f0, f1 = A[p], _mode(p, q, z1)
                    if (p, q, r) == (0, 0, 1):  # collapsed vertex
                        f0, f1 = one0, np.ones_like(z1)
                    elif (p, q) == (0, 1):      # collapsed edge
                        f0 = one0
                    rows.append(tensor(f0, f1, _mode(p + q, r, z2)))
    w = tensor(*(r[1] for r in rules))
    e0, e1, e2 = (tensor(*f) for f in ((z0, 0 * z1 + 1, 0 * z2 + 1), (one0, z1, 0 * z2 + 1),
                                       (one0, 0 * z1 + 1, z2)))
    C = np.zeros((3, 3, len(w)))
    C[2, 2] = 1
    if shape == "hex":
        C[0, 0] = C[1, 1] = 1
    elif shape == "prism":
        C[0, 0], C[0, 2], C[1, 1] = 2 / (1 - e2), (1 + e0) / (1 - e2), 1
    else:
        f = (1 - e1) * (1 - e2)
        C[0, 0], C[0, 1], C[0, 2] = 4 / f, 2 * (1 + e0) / f, 2 * (1 + e0) / f
        C[1, 1], C[1, 2] = 2 / (1 - e2), (1 + e1) / (1 - e2)

    def dev(a):
        return torch.as_tensor(np.ascontiguousarray(a), device="cuda")

    return dev(np.array(rows)), dev(w), [dev(r[2]) for r in rules], dev(C)


def _grad(u, Ds, nq):
    v = u.view(-1, nq[2], nq[1], nq[0])
    return torch.stack((v @ Ds[0].T, torch.einsum("jm,ekmi->ekji", Ds[1], v),
                        torch.einsum("km,emji->ekji", Ds[2], v))).view(3, *u.shape)


def _grad_t(g, Ds, nq):
    v = g.view(3, -1, nq[2], nq[1], nq[0])
    return (v[0] @ Ds[0] + torch.einsum("mj,ekmi->ekji", Ds[1], v[1])
            + torch.einsum("mk,emji->ekji", Ds[2], v[2])).reshape(g.shape[1:])


def _apply_exact(op, element, nq, jac, df, x, lam, vel):
    """One operator on a chunk of elements: jac (e, 1 or nt), df (9, e, 1 or nt),
    x (e, values)."""
    phi, w, Ds, C = element
    nt = w.numel()
    W = w * jac
    if op == "bwdtrans":
        return [x @ phi]
    if op == "iproduct":
        return [(W * x) @ phi.T]
    # R[a][k] = d eta_a / d x_k
    R = [[sum(C[a, j] * df[3 * k + j] for j in range(3)) for k in range(3)] for a in range(3)]
    if op == "physderiv":
        g = _grad(x, Ds, nq)
        return [sum(R[a][k] * g[a] for a in range(3)) for k in range(3)]
    if op == "iproduct_deriv":
        f = [W * v for v in x]
        v = torch.stack([sum(R[a][k] * f[k] for k in range(3)) for a in range(3)])
        return [_grad_t(v, Ds, nq) @ phi.T]
    u = x @ phi
    g = _grad(u, Ds, nq)
    dx = [sum(R[a][k] * g[a] for a in range(3)) for k in range(3)]
    v = torch.stack([sum(R[a][k] * (W * dx[k]) for k in range(3)) for a in range(3)])
    if op == "helmholtz":
        mass = lam * W * u
    else:
        mass = W * (sum(vel[k] * dx[k] for k in range(3)) - lam * u)
    return [(mass + _grad_t(v, Ds, nq)) @ phi.T]


def _exact_op(c, seed):
    jac, df, x, lam, vel = _inputs(c, seed)
    E, nt = c["elements"], _nt(c["shape"], c["nq"])
    element, nq = _element(c["shape"], c["nm"], c["nq"]), _points_per_direction(c["shape"], c["nq"])
    jac, df = jac.view(E, -1), df.view(9, E, -1)
    x = x.double()
    x = x.view(3, E, nt) if c["op"] == "iproduct_deriv" else x.view(E, -1)
    parts = []
    step = max(1, 2 ** 21 // nt)
    for e in range(0, E, step):
        s = slice(e, e + step)
        parts.append(_apply_exact(c["op"], element, nq, jac[s], df[:, s],
                                  x[:, s] if x.dim() == 3 else x[s], lam,
                                  None if vel is None else vel.view(3, E, nt)[:, s]))
    return [torch.cat([p[o] for p in parts]).ravel() for o in range(len(parts[0]))]


def _exact_solve(c, seed):
    """Conjugate gradients on the box to the limit of rounding."""
    b, lam = _solve_inputs(c, seed)
    n, nm = c["n"], c["nm"]
    P, nq = nm - 1, nm + 1
    element = _element("hex", nm, nq)
    z = torch.as_tensor(_rule(0, nq)[0], device="cuda")
    # curved map x + AMP sin sin sin of the box, elements ordered first direction fastest
    t = (torch.arange(n, device="cuda", dtype=torch.float64)[:, None] + (z + 1) / 2) / n
    X = [a.reshape(n ** 3, nq ** 3) for a in
         (t[None, None, :, None, None, :].expand(n, n, n, nq, nq, nq),
          t[None, :, None, None, :, None].expand(n, n, n, nq, nq, nq),
          t[:, None, None, :, None, None].expand(n, n, n, nq, nq, nq))]
    s, k = [torch.sin(math.pi * v) for v in X], [math.pi * torch.cos(math.pi * v) for v in X]
    dS = [k[0] * s[1] * s[2], s[0] * k[1] * s[2], s[0] * s[1] * k[2]]
    J = torch.stack([torch.stack([AMP * dS[l] + (r == l) for l in range(3)], -1)
                     for r in range(3)], -2) / (2 * n)
    jac = torch.linalg.det(J).abs()
    inv = torch.linalg.inv(J)  # [j, k] = d xi_j / d x_k
    df = torch.stack([inv[..., j, d] for d in range(3) for j in range(3)])
    # global numbers: vertex and interior modes along each direction
    line = torch.tensor([0, P] + list(range(1, P)), device="cuda")
    g = torch.arange(n, device="cuda")[:, None] * P + line
    N = n * P + 1
    gid = (g[:, None, None, :, None, None] * N * N + g[None, :, None, None, :, None] * N
           + g[None, None, :, None, None, :]).reshape(-1)
    inner = torch.zeros(N, dtype=torch.bool, device="cuda")
    inner[1:-1] = True
    free = (inner[:, None, None] & inner[None, :, None] & inner).reshape(-1).double()

    def assemble(v):
        # a sum in FP64 per global number
        return torch.zeros(N ** 3, dtype=torch.float64, device="cuda").index_add_(0, gid, v) * free

    def apply(v):
        y = _apply_exact("helmholtz", element, (nq,) * 3, jac, df, v[gid].view(n ** 3, -1), lam,
                         None)[0]
        return assemble(y.reshape(-1))

    r = assemble(b)
    phi2, W = element[0] ** 2, element[1] * jac
    M = 1 / (assemble(((W * inv.square().sum((-1, -2))) @ phi2.T).reshape(-1)) + 1e-30 + (1 - free))
    M = M / M.max()
    x, p, rz = torch.zeros_like(r), torch.zeros_like(r), None
    stop = 1e-28 * float(r @ r)
    for it in range(8000):
        zr = M * r
        new = r @ zr
        p = zr if rz is None else zr + (new / rz) * p
        rz = new
        Ap = apply(p)
        alpha = rz / (p @ Ap)
        x = x + alpha * p
        r = r - alpha * Ap
        if it % 50 == 0 and float(r @ r) < stop:
            break
    return x[gid]


def exact(case, seed):
    if case["kind"] == "op":
        return _exact_op(case, seed)
    if case["kind"] == "batch":
        parts = []
        for k, p in enumerate(_collections(case)):
            # a collection's three derivatives lie one after another
            parts += _exact_op(p, 1000 * seed + k)
        return torch.cat(parts)
    return _exact_solve(case, seed)
