"""Performance cases: the work a user of this package has it do, through its public entry points.

Kinds of case (every size is in the case itself):

axhelm        one application of the element operator, as the axhelm benchmark and a host
              code's own solver launch it: every order, one or three fields, Poisson (BK) or
              variable-coefficient Helmholtz, every precision, whole mesh or an element list.
apply         the assembled, masked operator of a problem (operator, gather-scatter, mask).
pcg           a whole linear solve on a box of perturbed trilinear hexahedra: the reference's
              algorithm in FP64 for a fixed number of iterations (the nekBone benchmark),
              mixed precision to a tolerance, or with the learned preconditioner.
net_forward   the learned preconditioner's network on element blocks.
net_gradient  loss and weight gradient of one training batch.
adv           the dealiased advection operator.
dot           the per-block partial sums of a weighted inner product.

Fields are uniform random numbers; the geometry is that of the meshes the package's own
benchmark uses (a box whose interior vertices are moved by up to a tenth of the spacing).
"""
import math
import os

import numpy as np
import torch

import nekbench_gb300 as nb

PRECISION = {"f64": nb.FP64, "f32": nb.FP32, "bf16": nb.BF16, "trilinear": nb.FP32_TRILINEAR,
             "split": nb.FP64_SPLIT}
# word sizes of (stored geometry and coefficients, vectors)
WORDS = {"f64": (8, 8), "split": (8, 8), "f32": (4, 4), "bf16": (2, 4), "trilinear": (0, 4)}
SHAPES = ((8, 16), (8, 8), (8, 4), (6, 16), (4, 16), (4, 8))  # (Nq, channels) the network is built for


def _axhelm(N, ex, ey, ez, fields=1, form="helmholtz", precision="f64", partial=False):
    return {"kind": "axhelm", "N": N, "ex": ex, "ey": ey, "ez": ez, "fields": fields, "form": form,
            "precision": precision, "partial": partial}


def _apply(N, ex, ey, ez, fields=1, form="helmholtz", precision="f64"):
    return {"kind": "apply", "N": N, "ex": ex, "ey": ey, "ez": ez, "fields": fields, "form": form,
            "precision": precision}


def _pcg(N, ex, ey, ez, solver, precond, form="helmholtz", fields=1, inner="f32", periodic=False,
         iterations=0, tol=1e-12):
    """iterations > 0: exactly that many; else to the relative residual tol."""
    return {"kind": "pcg", "N": N, "ex": ex, "ey": ey, "ez": ez, "solver": solver,
            "precond": precond, "form": form, "fields": fields, "inner": inner,
            "periodic": periodic, "iterations": iterations, "tol": tol}


def listed():
    return [
        # the reference's smallest operator benchmark: a mesh of 512 elements, launch bound
        dict(_axhelm(7, 8, 8, 8, form="poisson"), name="axhelm f64 poisson N7 E512"),
        # the headline: the operator over 134 million nodes
        dict(_axhelm(7, 64, 64, 64, form="poisson"), name="axhelm f64 poisson N7 E262144"),
        # the inner operators of a mixed-precision solve of a vector problem, at both orders of
        # that configuration, in its two storage forms
        dict(_axhelm(9, 32, 32, 32, fields=3, precision="f32"), name="axhelm f32 vector N9 E32768"),
        dict(_axhelm(7, 32, 32, 32, fields=3, precision="bf16"), name="axhelm bf16 vector N7 E32768"),
        # FP64 arrays in double-float arithmetic, the faster of the two FP64-accurate operators
        dict(_axhelm(7, 32, 32, 32, precision="split"), name="axhelm split N7 E32768"),
        # the assembled operator, as a caller's own Krylov loop applies it
        dict(_apply(7, 32, 32, 32, precision="f32"), name="apply f32 N7 E32768"),
        # nekBone's benchmark mode: periodic box, no preconditioner, a fixed number of iterations
        dict(_pcg(7, 16, 16, 32, "f64", "copy", form="poisson", periodic=True, iterations=100),
             name="pcg f64 poisson N7 E8192"),
        # a mixed-precision solve of the 4096-element configuration, small enough that launches count
        dict(_pcg(7, 16, 16, 16, "mixed", "jacobi"), name="pcg mixed N7 E4096"),
        # a solve with the learned preconditioner on the mesh it was trained on
        dict(_pcg(7, 24, 24, 24, "mixed", "learned"), name="pcg learned N7 E13824"),
        # one batch of the preconditioner's training, forward and backward, at its default size
        {"kind": "net_gradient", "Nq": 8, "channels": 16, "E": 4096, "name": "net gradient N7 C16 E4096"},
        # the dealiased advection benchmark at its default size
        {"kind": "adv", "N": 7, "cubN": 11, "E": 8192, "precision": "f64", "name": "adv f64 N7 cub11 E8192"},
        # the inner-product benchmark over the headline mesh's nodes
        {"kind": "dot", "variant": 0, "n": 64 ** 3 * 512, "fields": 1, "block": 256, "name": "dot v0 134M"},
    ]


def _box(rng, N, lo, hi):
    """Box counts with lo..hi nodes (log-uniform), sides of any parity."""
    E = max(1.0, math.exp(rng.uniform(math.log(lo), math.log(hi))) / (N + 1) ** 3)
    side = E ** (1 / 3)
    ex = max(1, round(side * rng.uniform(0.7, 1.4)))
    ey = max(1, round(side * rng.uniform(0.7, 1.4)))
    return ex, ey, max(1, round(E / (ex * ey)))


def draw(rng):
    kind = rng.choices(("axhelm", "apply", "pcg", "net", "adv", "dot"), (9, 2, 4, 2, 2, 1))[0]
    if kind in ("axhelm", "apply"):
        precision = rng.choices(("f64", "f32", "bf16", "trilinear", "split"), (4, 3, 2, 2, 2))[0]
        N = rng.randint(1, 13 if precision == "f64" else 11)
        fields = rng.choice((1, 1, 3))
        form = rng.choice(("poisson", "helmholtz"))
        if kind == "apply":
            return _apply(N, *_box(rng, N, 2e4, 2e7), fields, form, precision)
        partial = precision == "f64" and rng.random() < 0.25
        return _axhelm(N, *_box(rng, N, 2e4, 4e7), fields, form, precision, partial)
    if kind == "pcg":
        how = rng.choice(("f64", "split", "mixed", "mixed", "learned"))
        if how == "learned":
            return _pcg(7, *(rng.randint(5, 18) for _ in range(3)), "mixed", "learned")
        N = rng.randint(3, 9)
        most = max(5, 140 // (N + 1))
        box = tuple(rng.randint(4, most) for _ in range(3))
        if how == "mixed":
            return _pcg(N, *box, "mixed", "jacobi", fields=rng.choice((1, 1, 3)),
                        inner=rng.choice(("f32", "f32", "trilinear")))
        return _pcg(N, *box, how, "jacobi", fields=rng.choice((1, 3)), iterations=rng.randint(20, 100))
    if kind == "net":
        Nq, C = rng.choice(((8, 16),) * 3 + SHAPES)
        if rng.random() < 0.5:
            return {"kind": "net_forward", "Nq": Nq, "channels": C, "E": round(math.exp(rng.uniform(math.log(100), math.log(60000))))}
        return {"kind": "net_gradient", "Nq": Nq, "channels": C, "E": round(math.exp(rng.uniform(math.log(100), math.log(6000))))}
    if kind == "adv":
        N = rng.randint(2, 9)
        cub = rng.choice((N, math.ceil(1.5 * (N + 1)) - 1))
        E = max(1, round(math.exp(rng.uniform(math.log(2e4), math.log(4e6))) / (N + 1) ** 3))
        return {"kind": "adv", "N": N, "cubN": cub, "E": E, "precision": rng.choice(("f64", "split"))}
    variant = rng.choice((0, 1, 2))
    return {"kind": "dot", "variant": variant, "n": round(math.exp(rng.uniform(math.log(2e4), math.log(1e8)))),
            "fields": rng.choice((1, 3)) if variant == 2 else 1,
            "block": 256 if variant == 1 else rng.choice((256, 512, 1024))}


# --------------------------------------------------------------------------- inputs (plain torch and numpy)
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rand(g, n, lo, hi, dtype=torch.float64):
    return torch.empty(n, dtype=dtype, device="cuda").uniform_(lo, hi, generator=g)


def _gll(N):
    """Gauss-Lobatto-Legendre nodes and weights of order N."""
    P = np.polynomial.legendre.Legendre.basis(N)
    inner = np.sort(P.deriv().roots().real) if N > 1 else np.zeros(0)
    for _ in range(3):  # Newton on P_N' (its second derivative from Legendre's equation)
        d1, p = P.deriv()(inner), P(inner)
        inner = inner - d1 * (1 - inner ** 2) / (2 * inner * d1 - N * (N + 1) * p)
    x = np.concatenate([[-1.0], inner, [1.0]])
    x = 0.5 * (x - x[::-1])
    return x, 2.0 / (N * (N + 1) * P(x) ** 2)


def _lagrange(x):
    return np.array([1.0 / np.prod([x[j] - x[k] for k in range(len(x)) if k != j]) for j in range(len(x))])


def _deriv(x):
    """D[i, m] = derivative of the m-th Lagrange polynomial at node i."""
    lam = _lagrange(x)
    D = np.array([[0.0 if i == m else lam[m] / (lam[i] * (x[i] - x[m])) for m in range(len(x))]
                  for i in range(len(x))])
    return D - np.diag(D.sum(1))


def _interp(x, y):
    """I[i, a] = a-th Lagrange polynomial of the nodes x at y[i]."""
    lam = _lagrange(x)
    rows = []
    for t in y:
        d = t - x
        if np.min(np.abs(d)) < 1e-14:
            rows.append((np.abs(d) < 1e-14).astype(float))
        else:
            rows.append(lam / d / np.sum(lam / d))
    return np.array(rows)


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _elements(c):
    return c["ex"] * c["ey"] * c["ez"]


def _vertices(c, seed):
    """[3][E, 8] element vertices (r fastest, then s, t with the corners of each face in
    cyclic order) of the unit box with moved interior vertices."""
    n = (c["ex"], c["ey"], c["ez"])
    g = _gen(seed * 7919 + 1)
    grid = torch.meshgrid(*[torch.arange(m + 1, device="cuda", dtype=torch.float64) / m for m in n[::-1]],
                          indexing="ij")
    inside = torch.ones(grid[0].shape, dtype=torch.bool, device="cuda")
    if not c.get("periodic"):
        for d in range(3):
            inside &= (grid[d] > 0) & (grid[d] < 1)
        move = [_rand(g, grid[0].numel(), -0.1, 0.1).view(grid[0].shape) for _ in range(3)]
    else:
        move = [torch.zeros_like(grid[0]) for _ in range(3)]
    out = []
    for d in range(3):  # x varies along the last axis of the grid
        v = grid[2 - d] + torch.where(inside, move[d] / n[d], torch.zeros_like(move[d]))
        corner = [v[k:k + n[2], j:j + n[1], i:i + n[0]].reshape(-1)
                  for k in (0, 1) for j, i in ((0, 0), (0, 1), (1, 1), (1, 0))]
        out.append(torch.stack(corner, 1).contiguous())
    return out


_SIGNS = [(-1, -1, -1), (1, -1, -1), (1, 1, -1), (-1, 1, -1), (-1, -1, 1), (1, -1, 1), (1, 1, 1), (-1, 1, 1)]


def _coefficients(V):
    """[E, 3, 8]: x(r,s,t) in the basis {1, r, s, t, rs, rt, st, rst}."""
    B = torch.tensor([[1, r, s, t, r * s, r * t, s * t, r * s * t] for r, s, t in _SIGNS],
                     dtype=torch.float64, device="cuda") * 0.125
    return torch.stack([v @ B for v in V], 1)


def _factors(coef, N):
    """[E, 7, Nq^3]: GWJ, G00, G01, G02, G11, G12, G22 from trilinear coefficients (float64)."""
    x, w = (_cuda(a) for a in _gll(N))
    r, s, t = x.view(1, 1, 1, -1), x.view(1, 1, -1, 1), x.view(1, -1, 1, 1)
    a = coef.double().view(-1, 3, 8, 1, 1, 1)
    J = [[a[:, c, 1] + a[:, c, 4] * s + a[:, c, 5] * t + a[:, c, 7] * (s * t),
          a[:, c, 2] + a[:, c, 4] * r + a[:, c, 6] * t + a[:, c, 7] * (r * t),
          a[:, c, 3] + a[:, c, 5] * r + a[:, c, 6] * s + a[:, c, 7] * (r * s)] for c in range(3)]

    def cross(p, q):
        u, v = [J[c][p] for c in range(3)], [J[c][q] for c in range(3)]
        return u[1] * v[2] - u[2] * v[1], u[2] * v[0] - u[0] * v[2], u[0] * v[1] - u[1] * v[0]
    gr, gs, gt = cross(1, 2), cross(2, 0), cross(0, 1)
    det = sum(J[c][0] * gr[c] for c in range(3))
    W = w.view(1, 1, 1, -1) * w.view(1, 1, -1, 1) * w.view(1, -1, 1, 1)
    wi = W / det

    def dot(p, q):
        return wi * (p[0] * q[0] + p[1] * q[1] + p[2] * q[2])
    shape = det.shape
    return torch.stack([v.expand(shape) for v in (det * W, dot(gr, gr), dot(gr, gs), dot(gr, gt),
                                                  dot(gs, gs), dot(gs, gt), dot(gt, gt))], 1).reshape(shape[0], 7, -1)


def _geometry(coef, N, dtype):
    E, Np = coef.shape[0], (N + 1) ** 3
    out = torch.empty(E, 7, Np, dtype=dtype, device="cuda")
    step = max(1, (1 << 23) // Np)
    for e in range(0, E, step):
        out[e:e + step] = _factors(coef[e:e + step], N)
    return out


def _global_ids(c):
    """[E*Np] global node numbers from 1 and, on a box with a boundary, the boundary nodes."""
    n, N = (c["ex"], c["ey"], c["ez"]), c["N"]
    axis = []
    for m in n:
        a = torch.arange(m, device="cuda").view(-1, 1) * N + torch.arange(N + 1, device="cuda").view(1, -1)
        axis.append(a % (m * N) if c.get("periodic") else a)
    size = [m * N if c.get("periodic") else m * N + 1 for m in n]
    i = axis[0].view(1, 1, n[0], 1, 1, N + 1)
    j = axis[1].view(1, n[1], 1, 1, N + 1, 1)
    k = axis[2].view(n[2], 1, 1, N + 1, 1, 1)
    shape = (n[2], n[1], n[0], N + 1, N + 1, N + 1)
    ids = (1 + i + size[0] * (j + size[1] * k)).expand(shape).reshape(-1)
    if c.get("periodic"):
        return ids, None, size
    edge = torch.zeros(shape, dtype=torch.bool, device="cuda")
    for a, s in zip((i, j, k), size):
        edge |= ((a == 0) | (a == s - 1)).expand(shape)
    return ids, edge.reshape(-1), size


def _problem(c, seed):
    """Mesh, coefficients and a right-hand side that is one value per global node."""
    V = _vertices(c, seed)
    ids, edge, size = _global_ids(c)
    g = _gen(seed * 7919 + 2)
    L, f = ids.numel(), c["fields"]
    lam = None
    if c["form"] == "helmholtz":
        if c.get("precond") == "learned":  # the smooth coefficients the network was trained for
            k = torch.randint(1, 5, (3,), generator=torch.Generator().manual_seed(int(seed))).tolist()
            x, y, z = _nodes(_coefficients(V), c["N"])
            lam = torch.cat([torch.ones(L, dtype=torch.float64, device="cuda"),
                             1 + 0.5 * torch.sin(2 * math.pi * (k[0] * x + k[1] * y + k[2] * z))])
        else:
            lam = torch.cat([_rand(g, L, 0.5, 1.5), _rand(g, L, 0.5, 2.0)])
    b = []
    for _ in range(f):
        v = _rand(g, size[0] * size[1] * size[2], -1, 1)
        if edge is None:
            v = v - v.mean()
        b.append(v[ids - 1] if edge is None else torch.where(edge, 0.0, v[ids - 1]))
    return V, ids, edge, lam, torch.cat(b)


def _nodes(coef, N):
    x = _cuda(_gll(N)[0])
    r, s, t = x.view(1, 1, 1, -1), x.view(1, 1, -1, 1), x.view(1, -1, 1, 1)
    a = coef.view(-1, 3, 8, 1, 1, 1)
    return [(a[:, c, 0] + a[:, c, 1] * r + a[:, c, 2] * s + a[:, c, 3] * t + a[:, c, 4] * (r * s)
             + a[:, c, 5] * (r * t) + a[:, c, 6] * (s * t) + a[:, c, 7] * (r * s * t)).reshape(-1) for c in range(3)]


def _handle(c, V, ids, edge):
    """The problem handle a program keeps, on its own mesh."""
    N = c["N"]
    gids = ids if edge is None else torch.where(edge, 0, ids)
    mask = None if edge is None else torch.nonzero(edge).view(-1).int().cpu().numpy()
    ggeo = _geometry(_coefficients(V), N, torch.float64).reshape(-1)
    v = [a.reshape(-1).cpu().numpy() for a in V]
    bp = nb.BP.from_mesh(N, _elements(c), ggeo, gids.cpu().numpy(), mask, *v, Nfields=c["fields"])
    bp._keep = None  # the handle holds its own copies
    return bp


def _axhelm_inputs(c, seed):
    E, Np, N = _elements(c), (c["N"] + 1) ** 3, c["N"]
    store = {"f64": torch.float64, "split": torch.float64, "f32": torch.float32, "bf16": torch.bfloat16,
             "trilinear": torch.float32}[c["precision"]]
    vec = torch.float64 if WORDS[c["precision"]][1] == 8 else torch.float32
    coef = _coefficients(_vertices(c, seed))
    geo = coef.float().reshape(-1) if c["precision"] == "trilinear" else _geometry(coef, N, store).view(-1)
    g = _gen(seed * 7919 + 3)
    lam = None
    if c["form"] == "helmholtz":
        lam = torch.cat([_rand(g, E * Np, 0.5, 1.5, vec), _rand(g, E * Np, 0.5, 2.0, vec)]).to(store)
    q = _rand(g, c["fields"] * E * Np, -1, 1, vec)
    elements = None
    if c.get("partial"):  # about half of the elements, in ascending order, as a halo split lists them
        elements = torch.nonzero(_rand(g, E, 0, 1) < 0.5).view(-1).int()
        if elements.numel() == 0:
            elements = torch.zeros(1, dtype=torch.int32, device="cuda")
    return geo, lam, q, _cuda(_deriv(_gll(N)[0])).to(vec).reshape(-1), elements


def _net_inputs(c, seed):
    g = _gen(seed * 7919 + 4)
    C, Np = c["channels"], c["Nq"] ** 3
    bound = np.concatenate([np.full(27 * C, math.sqrt(6 / 27)), np.full(27 * C * C, math.sqrt(6 / (27 * C))),
                            np.full(27 * C, 0.1 * math.sqrt(6 / (27 * C)))])
    w = (_rand(g, bound.size, -1, 1) * _cuda(bound)).float()
    x = torch.randn(c["E"] * Np, device="cuda", generator=g)
    y = 0.3 * torch.randn(c["E"] * Np, device="cuda", generator=g)
    return w, x, y


def _adv_inputs(c, seed):
    g = _gen(seed * 7919 + 5)
    Nq, cq, E = c["N"] + 1, c["cubN"] + 1, c["E"]
    x, y = _gll(c["N"])[0], _gll(c["cubN"])[0]
    vgeo = _rand(g, 12 * E * Nq ** 3, 0.5, 1.5)
    cubvgeo = _rand(g, 12 * E * cq ** 3, 0.5, 1.5)
    D, I = _cuda(_deriv(y)), _cuda(_interp(x, y))  # I[i, a]; the operator takes its transpose
    U = _rand(g, 3 * E * Nq ** 3, -1, 1)
    return vgeo, cubvgeo, D.reshape(-1), I.t().contiguous().reshape(-1), U


# --------------------------------------------------------------------------- the package's side
def prepare(case, seed):
    c, s = case, {"case": case}
    if c["kind"] == "axhelm":
        geo, lam, q, D, elements = _axhelm_inputs(c, seed)
        name = "axhelm" + ("Partial" if c["partial"] else "") + ("_bk" if c["form"] == "poisson" else "") + \
            ("_n3" if c["fields"] == 3 else "") + "_v0"
        E = _elements(c) if elements is None else elements.numel()
        args = (E, _elements(c) * (c["N"] + 1) ** 3) + (() if elements is None else (elements,)) + (geo, D, lam, q)
        s.update(kernel=nb.load_ax_kernel(name, c["N"], PRECISION[c["precision"]]), args=args, Aq=torch.zeros_like(q))
    elif c["kind"] in ("apply", "pcg"):
        V, ids, edge, lam, b = _problem(c, seed)
        s.update(bp=_handle(c, V, ids, edge), lam=lam)
        if c["kind"] == "apply":
            store, vec = {"f64": (torch.float64,) * 2, "split": (torch.float64,) * 2, "f32": (torch.float32,) * 2,
                          "bf16": (torch.bfloat16, torch.float32), "trilinear": (torch.float32,) * 2}[c["precision"]]
            s.update(lam=None if lam is None else lam.to(store), q=b.to(vec), Aq=torch.zeros_like(b, dtype=vec))
        else:
            s.update(b=b, r=torch.empty_like(b), x=torch.empty_like(b), net=None)
            if c["precond"] == "learned":
                s["net"] = nb.Net.load(os.path.join(os.path.dirname(nb.__file__), "weights", "precond_n7_c16.bin"))
    elif c["kind"] in ("net_forward", "net_gradient"):
        w, x, y = _net_inputs(c, seed)
        net = nb.Net(c["Nq"], c["channels"], 3)
        net.set_weights(w.cpu().numpy())
        s.update(net=net, x=x, y=y, out=torch.zeros_like(x))
    elif c["kind"] == "adv":
        vgeo, cubvgeo, D, It, U = _adv_inputs(c, seed)
        s.update(kernel=nb.load_adv_kernel(c["N"], c["cubN"], PRECISION[c["precision"]]), NU=torch.zeros_like(U),
                 args=(c["E"], vgeo, cubvgeo, D, It, c["E"] * (c["N"] + 1) ** 3, U))
    else:
        g = _gen(seed * 7919 + 6)
        n, f = c["n"], c["fields"]
        name = ("weightedInnerProduct2_v0", "weightedInnerProduct2_v1", "weightedBlockInnerProduct2")[c["variant"]]
        w, x, y = _rand(g, n, 0, 1), _rand(g, f * n, -1, 1), _rand(g, f * n, -1, 1)
        out = torch.zeros(nb.dot_num_blocks(n, c["block"]), dtype=torch.float64, device="cuda")
        s.update(kernel=nb.load_dot_kernel(name, c["block"], f), out=out,
                 args=((n, n) if c["variant"] == 2 else (n,)) + (w, x, y))
    return s


_SOLVER = {"f64": nb.SOLVER_FP64, "split": nb.SOLVER_FP64_SPLIT, "mixed": nb.SOLVER_MIXED}
_PRECOND = {"copy": nb.PRECOND_COPY, "jacobi": nb.PRECOND_JACOBI, "learned": nb.PRECOND_LEARNED}


def run(s):
    c = s["case"]
    if c["kind"] == "axhelm":
        s["kernel"](*s["args"], s["Aq"])
        return s["Aq"]
    if c["kind"] == "apply":
        s["bp"].apply(s["q"], s["Aq"], s["lam"], c["form"] == "poisson", PRECISION[c["precision"]])
        return s["Aq"]
    if c["kind"] == "pcg":
        s["r"].copy_(s["b"])  # the solver overwrites its right-hand side and its guess
        s["x"].zero_()
        s["bp"].pcg(s["lam"], s["r"], s["x"], c["tol"], c["iterations"] or 20000, solver=_SOLVER[c["solver"]],
                    precond=_PRECOND[c["precond"]], fixed_iterations=c["iterations"] > 0,
                    bk=c["form"] == "poisson", inner_precision=PRECISION[c["inner"]], net=s["net"])
        return s["x"]
    if c["kind"] == "net_forward":
        s["net"].forward(s["x"], s["out"], c["E"])
        return s["out"]
    if c["kind"] == "net_gradient":
        gradient, loss = s["net"].gradient(s["x"], s["y"], c["E"])
        return {"gradient": gradient, "loss": loss}
    if c["kind"] == "adv":
        s["kernel"](*s["args"], s["NU"])
        return s["NU"]
    s["kernel"](*s["args"], s["out"])
    return s["out"]


# --------------------------------------------------------------------------- what a pass cannot do without
def _operator_work(c, precision, E):
    """Each stored factor, coefficient and input value read once, each output written once."""
    Nq, f = c["N"] + 1, c["fields"]
    geo, vec = WORDS[precision]
    nodes = E * Nq ** 3
    helm = c["form"] == "helmholtz"
    stored = 96 * E if precision == "trilinear" else (7 if helm else 6) * geo * nodes
    lam = 2 * (geo or vec) * nodes if helm else 0
    flops = nodes * (f * (12 * Nq + 15 + (5 if helm else 0)))
    return stored + lam + 2 * f * vec * nodes, flops


def work(case):
    c = case
    if c["kind"] in ("axhelm", "apply"):
        E = _elements(c) // 2 if c.get("partial") else _elements(c)
        b, fl = _operator_work(c, c["precision"], max(E, 1))
        return {"bytes": b, "flops": fl}
    if c["kind"] == "pcg":
        precision = c["inner"] if c["solver"] == "mixed" else c["solver"]
        n = c["iterations"] or 7 * c["N"] * max(c["ex"], c["ey"], c["ez"])  # measured counts lie near this
        b, fl = _operator_work(c, precision, _elements(c))
        nodes, vec = _elements(c) * (c["N"] + 1) ** 3, WORDS[precision][1]
        # per iteration beside the operator: read and write x, r, p; read A p, the weights and the diagonal
        b += vec * nodes * (7 * c["fields"] + 2)
        fl += 14 * nodes * c["fields"]
        if c["precond"] == "learned":
            fl += 15552 * nodes
        return {"bytes": n * b, "flops": n * fl}
    if c["kind"] in ("net_forward", "net_gradient"):
        C, nodes = c["channels"], c["E"] * c["Nq"] ** 3
        macs = 27 * C * (C + 2)
        return {"bytes": 8 * nodes + 8 * macs, "flops": nodes * macs * (2 if c["kind"] == "net_forward" else 6)}
    if c["kind"] == "adv":
        n, q = c["N"] + 1, c["cubN"] + 1
        tensor = n ** 3 * q + n ** 2 * q ** 2 + n * q ** 3
        return {"bytes": 8 * c["E"] * (10 * q ** 3 + 7 * n ** 3),
                "flops": c["E"] * (12 * tensor + 18 * q ** 4 + 33 * q ** 3 + 3 * n ** 3)}
    return {"bytes": 8 * (c["n"] * (1 + 2 * c["fields"]) + c["n"] // c["block"]), "flops": 3 * c["n"] * c["fields"]}


# --------------------------------------------------------------------------- the same in 64 bits, plain torch
def _element_operator(G, D, q, lam0, lam1):
    """q [E, n, n, n]; G [E, 7, n, n, n]; A q of each element, before assembly."""
    def along(M, v, d):  # sum_m M[i, m] v[.., m, ..] along axis d
        return torch.movedim(torch.movedim(v, d, -1) @ M.t(), -1, d)
    qr, qs, qt = along(D, q, 3), along(D, q, 2), along(D, q, 1)
    gr = G[:, 1] * qr + G[:, 2] * qs + G[:, 3] * qt
    gs = G[:, 2] * qr + G[:, 4] * qs + G[:, 5] * qt
    gt = G[:, 3] * qr + G[:, 5] * qs + G[:, 6] * qt
    if lam0 is not None:
        gr, gs, gt = lam0 * gr, lam0 * gs, lam0 * gt
    out = along(D.t(), gr, 3) + along(D.t(), gs, 2) + along(D.t(), gt, 1)
    return out if lam1 is None else out + G[:, 0] * lam1 * q


def _exact_axhelm(c, seed):
    geo, lam, q, D, elements = _axhelm_inputs(c, seed)
    n, E = c["N"] + 1, _elements(c)
    D = D.double().view(n, n)
    cube = (E, n, n, n)
    lam = [None, None] if lam is None else [v.view(cube) for v in lam.view(2, -1)]
    out = torch.zeros(c["fields"], *cube, dtype=torch.float64, device="cuda")
    step = max(1, (1 << 23) // n ** 3)
    for e in range(0, E, step):
        s = slice(e, e + step)
        if c["precision"] == "trilinear":
            G = _factors(geo.view(E, 3, 8)[s], c["N"]).view(-1, 7, n, n, n)
        else:
            G = geo.view(E, 7, n, n, n)[s].double()
        l0, l1 = (None if v is None else v[s].double() for v in lam)
        for f in range(c["fields"]):
            out[f, s] = _element_operator(G, D, q.view(c["fields"], *cube)[f, s].double(), l0, l1)
    if elements is not None:
        keep = torch.zeros(E, dtype=torch.bool, device="cuda")
        keep[elements.long()] = True
        out[:, ~keep] = 0
    return out.view(-1)


class _Assembled:
    """mask(gs(operator)) with the problem's own coefficients, FP64."""

    def __init__(self, c, seed, lam=None, store=torch.float64):
        V, self.ids, self.edge, l, self.b = _problem(c, seed)
        lam = l if lam is None else lam
        n, E = c["N"] + 1, _elements(c)
        self.cube, self.f, self.c = (E, n, n, n), c["fields"], c
        coef = _coefficients(V)
        if c.get("precision") == "trilinear":
            coef = coef.float()
        self.G = _geometry(coef, c["N"], torch.float64).to(store).double().view(E, 7, n, n, n)
        D = _cuda(_deriv(_gll(c["N"])[0]))
        self.D = D.float().double() if c.get("precision") in ("f32", "bf16", "trilinear") else D
        self.lam = [None, None] if lam is None else [v.to(store).double().view(self.cube) for v in lam.view(2, -1)]
        count = torch.zeros(int(self.ids.max()) + 1, dtype=torch.float64, device="cuda")
        self.w = 1 / count.index_add_(0, self.ids, torch.ones_like(self.ids, dtype=torch.float64))[self.ids]

    def gs(self, v):
        total = torch.zeros(int(self.ids.max()) + 1, dtype=torch.float64, device="cuda").index_add_(0, self.ids, v)
        out = total[self.ids]
        return out if self.edge is None else torch.where(self.edge, 0.0, out)

    def __call__(self, v):
        out = []
        for x in v.view(self.f, -1):
            y = torch.empty(self.cube, dtype=torch.float64, device="cuda")
            x, step = x.view(self.cube), max(1, (1 << 23) // self.cube[1] ** 3)
            for e in range(0, self.cube[0], step):
                s = slice(e, e + step)
                y[s] = _element_operator(self.G[s], self.D, x[s], *(None if a is None else a[s] for a in self.lam))
            out.append(self.gs(y.view(-1)))
        return torch.cat(out)

    def diagonal(self):
        G, D, out = self.G, self.D ** 2, torch.zeros(self.cube, dtype=torch.float64, device="cuda")
        l0 = 1.0 if self.lam[0] is None else self.lam[0]
        for slot, d in ((1, 3), (4, 2), (6, 1)):
            out += torch.movedim(torch.movedim(l0 * G[:, slot], d, -1) @ D, -1, d)
        dd = torch.diagonal(self.D)
        r, s, t = dd.view(1, 1, 1, -1), dd.view(1, 1, -1, 1), dd.view(1, -1, 1, 1)
        out += 2 * l0 * (G[:, 2] * r * s + G[:, 3] * r * t + G[:, 5] * s * t)
        if self.lam[1] is not None:
            out += G[:, 0] * self.lam[1]
        total = self.gs(out.view(-1))
        return total if self.edge is None else torch.where(self.edge, 1.0, total)


def _exact_apply(c, seed):
    store = {"f32": torch.float32, "bf16": torch.bfloat16}.get(c["precision"], torch.float64)
    A = _Assembled(c, seed, store=store)
    if c["precision"] == "trilinear" and A.lam[0] is not None:
        A.lam = [v.float().double() for v in A.lam]
    b = A.b if WORDS[c["precision"]][1] == 8 else A.b.float().double()
    return A(b)


def _exact_pcg(c, seed):
    A = _Assembled(c, seed)
    nodes = A.b.numel()
    if nodes * (c["iterations"] or 900) > 1.2e10:
        return None
    inv = 1 / A.diagonal().repeat(c["fields"]) if c["precond"] != "copy" else torch.ones_like(A.b)
    w = A.w.repeat(c["fields"])
    r, x = A.b.clone(), torch.zeros_like(A.b)
    z = inv * r
    p, rz, r0 = z.clone(), (w * r * z).sum(), (w * r * r).sum()
    for k in range(c["iterations"] or 20000):
        Ap = A(p)
        alpha = rz / (w * p * Ap).sum()
        x += alpha * p
        r -= alpha * Ap
        z = inv * r
        rz, old = (w * r * z).sum(), rz
        p = z + (rz / old) * p
        if not c["iterations"] and k % 16 == 0 and (w * r * r).sum() <= 1e-26 * r0:
            break
    return x


def _conv(x, w):
    """3x3x3 convolution with zero padding, x [E, ci, n, n, n], w [co, ci, 3, 3, 3], float64."""
    n = x.shape[-1]
    p = torch.nn.functional.pad(x, (1,) * 6)
    out = 0
    for k in range(3):
        for j in range(3):
            for i in range(3):
                out = out + torch.einsum("ecxyz,oc->eoxyz", p[:, :, k:k + n, j:j + n, i:i + n], w[:, :, k, j, i])
    return out


def _network(x, w, C):
    w1, w2, w3 = torch.split(w, (27 * C, 27 * C * C, 27 * C))
    gelu = lambda v: 0.5 * v * (1 + torch.tanh(0.7978845608028654 * (v + 0.044715 * v ** 3)))  # noqa: E731
    h = gelu(_conv(x, w1.view(C, 1, 3, 3, 3)))
    h = gelu(_conv(h, w2.view(C, C, 3, 3, 3)))
    return _conv(h, w3.view(1, C, 3, 3, 3))


def _exact_net(c, seed):
    w, x, y = _net_inputs(c, seed)
    n, E, C = c["Nq"], c["E"], c["channels"]
    x, y = x.double().view(E, 1, n, n, n), y.double().view(E, 1, n, n, n)
    if c["kind"] == "net_forward":  # the network's weights are BF16
        w = w.bfloat16().double()
        with torch.no_grad():
            return torch.cat([_network(x[e:e + 2048], w, C) for e in range(0, E, 2048)]).view(-1)
    w = w.double().requires_grad_()
    loss = 0.0
    for e in range(0, E, 512):
        part = ((_network(x[e:e + 512], w, C) - y[e:e + 512]) ** 2).sum() / (E * n ** 3)
        part.backward()
        loss += float(part.detach())
    return {"gradient": w.grad.cpu().numpy(), "loss": loss}


def _exact_adv(c, seed):
    vgeo, cubvgeo, D, It, U = _adv_inputs(c, seed)
    n, q, E = c["N"] + 1, c["cubN"] + 1, c["E"]
    D, I = D.view(q, q), It.view(n, q).t()
    out = torch.empty(3, E, n, n, n, dtype=torch.float64, device="cuda")
    step = max(1, (1 << 22) // q ** 3)

    def all3(M, v):
        for d in (-1, -2, -3):
            v = torch.movedim(torch.movedim(v, d, -1) @ M.t(), -1, d)
        return v
    for e in range(0, E, step):
        s = slice(e, e + step)
        Uc = all3(I, U.view(3, E, n, n, n)[:, s])
        m = cubvgeo.view(E, 12, q, q, q)[s]
        jw = m[:, 5]
        rows = ((0, 1, 7), (2, 3, 8), (9, 10, 11))  # metric slots of grad r, grad s, grad t
        hat = [jw * sum(m[:, a] * Uc[d] for d, a in enumerate(row)) for row in rows]
        for f in range(3):
            grad = [torch.movedim(torch.movedim(Uc[f], d, -1) @ D.t(), -1, d) for d in (-1, -2, -3)]
            out[f, s] = all3(I.t(), sum(h * g for h, g in zip(hat, grad))) * vgeo.view(E, 12, n, n, n)[s, 6]
    return out.view(-1)


def _exact_dot(c, seed):
    g = _gen(seed * 7919 + 6)
    n, f = c["n"], c["fields"]
    w, x, y = _rand(g, n, 0, 1), _rand(g, f * n, -1, 1), _rand(g, f * n, -1, 1)
    v = (w * (x * y).view(f, n)).sum(0)
    return torch.nn.functional.pad(v, (0, -n % c["block"])).view(-1, c["block"]).sum(1)


def exact(case, seed):
    kind = case["kind"]
    how = {"axhelm": _exact_axhelm, "apply": _exact_apply, "pcg": _exact_pcg, "net_forward": _exact_net,
           "net_gradient": _exact_net, "adv": _exact_adv, "dot": _exact_dot}[kind]
    return how(case, seed)
