"""Performance cases of the H2 single-layer operator: products, assemblies and
whole solves, through the package's public entry points.

A case is one of three kinds of work that a boundary-element program does:

product   y = A x with the assembled operator, device tensors in and out: the
          step of a Krylov method that the program runs itself.
assemble  DiscreteOperator.compute() (near-field quadrature and far-field
          couplings) for a geometry, for Helmholtz at a wavenumber the operator
          has not been assembled at, then the first product with it.
solve     the whole call of the examples: load vectors of analytic data, the
          batched solve to the tolerance, the potential at points off the
          surface (the density itself is known only to the condition number
          times the tolerance; the potential is what such a program is after).

Geometries are the two spheres and the torus of the repository's benchmark
and tests: "cube" the analytic cube sphere, "sphere" and "torus" the Bezier
patches of tests/golden/geo.
"""
import functools
import math
import os

import numpy as np
import torch

import bembel_gb300 as bg

GEO = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tests", "golden", "geo")
PATCHES = {"cube": 6, "sphere": 6, "torus": 16}
SOLVE_TOL = 1e-8
MAX_EXACT_ELEMENTS = 1600  # the dense product of exact() stays within seconds


def _case(work, operator, geometry, M, P, n_p, nrhs, precision, kappa=0.0, name=None):
    c = {"work": work, "operator": operator, "geometry": geometry, "M": M, "P": P, "n_p": n_p, "nrhs": nrhs,
         "precision": precision, "kappa": kappa}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: one product of a few hundred unknowns, where launches and latency count
        _case("product", "laplace", "cube", 2, 1, 6, 1, "fp64", name="product_laplace_M2_1_fp64"),
        # one vector at a time on an ordinary size, as an unbatched Krylov solver of the user's applies it
        _case("product", "laplace", "sphere", 4, 2, 9, 1, "fp64", name="product_laplace_M4_1_fp64"),
        # the benchmark's operator, a full batch of vectors, at either precision it is quoted at
        _case("product", "laplace", "sphere", 5, 2, 9, 32, "fp64", name="product_laplace_M5_32_fp64"),
        _case("product", "laplace", "sphere", 5, 2, 9, 32, "mixed", name="product_laplace_M5_32_mixed"),
        # complex operators: scalar on the torus with the sweep's interpolation degree, and the vector-valued EFIE
        _case("product", "helmholtz", "torus", 3, 2, 10, 16, "mixed", 3.0, name="product_helmholtz_M3_16_mixed"),
        _case("product", "maxwell", "sphere", 3, 2, 9, 5, "fp64", 2.0, name="product_maxwell_M3_5_fp64"),
        # assembly: once per geometry for Laplace, once per wavenumber of a sweep for Helmholtz
        _case("assemble", "laplace", "sphere", 4, 2, 9, 1, "fp64", name="assemble_laplace_M4"),
        _case("assemble", "helmholtz", "torus", 3, 2, 10, 1, "fp64", 3.0, name="assemble_helmholtz_M3"),
        # whole calls: the plain example (one right-hand side, FP64), the benchmark's batched mixed solve,
        # and the complex workloads with the solver's FP32 inner operator
        _case("solve", "laplace", "cube", 3, 1, 6, 1, "fp64", name="solve_laplace_M3_1_fp64"),
        _case("solve", "laplace", "sphere", 5, 2, 9, 32, "mixed", name="solve_laplace_M5_32_mixed"),
        _case("solve", "helmholtz", "torus", 3, 2, 10, 16, "fp32", 2.0, name="solve_helmholtz_M3_16_fp32"),
        _case("solve", "maxwell", "sphere", 3, 2, 9, 8, "fp32", 2.0, name="solve_maxwell_M3_8_fp32"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    """A case of the same ranges: refinement levels, both degrees, every operator, geometry and precision,
    odd interpolation degrees and column counts (products also past the 32 columns of one batch)."""
    work = rng.choice(["product", "product", "product", "assemble", "solve"])
    operator = rng.choice(["laplace", "laplace", "helmholtz", "maxwell"] if work != "assemble" else
                          ["laplace", "helmholtz"])
    geometry = rng.choice(["cube", "sphere", "torus"])
    P = rng.choice([1, 2])
    precision = rng.choice(["fp64", "mixed", "fp32"]) if work != "assemble" else "fp64"
    top = {"laplace": 5, "helmholtz": 4, "maxwell": 3}[operator]
    if work == "assemble" or (work == "solve" and operator == "laplace"):
        top -= 1
    if work == "solve" and (operator != "laplace" or precision == "fp64"):
        top = 3
    M = rng.randint(2, top)
    if geometry == "torus":
        M = max(2, M - 1)
    kappa = round(rng.uniform(0.5, 4.0 if operator == "helmholtz" else 2.0), 3) if operator != "laplace" else 0.0
    n_p = rng.randint(6, 9) if operator == "laplace" else rng.randint(7, 10 if operator == "helmholtz" else 9)
    most = 45 if work == "product" and M < 5 else 32
    if operator != "laplace":
        most = 20 if work == "product" else 12
    return _case(work, operator, geometry, M, P, n_p, 1 if work == "assemble" else _log_int(rng, 1, most), precision,
                 kappa)


def _operator(case, kappa, context=None):
    geo = (bg.Geometry.cube_sphere(context) if case["geometry"] == "cube" else
           bg.Geometry(os.path.join(GEO, case["geometry"] + ".dat"), context))
    lin = {"laplace": bg.LaplaceSingleLayerOperator, "helmholtz": bg.HelmholtzSingleLayerOperator,
           "maxwell": bg.MaxwellSingleLayerOperator}[case["operator"]]()
    if lin.is_complex:
        lin.set_wavenumber(kappa)
    return bg.DiscreteOperator(bg.AnsatzSpace(geo, case["M"], case["P"]), lin, n_p=case["n_p"])


def _wavenumber(case, seed):
    """The wavenumber: fixed for an operator in hand, near the case's for an assembly (a sweep's next one)."""
    if case["work"] != "assemble" or not case["kappa"]:
        return case["kappa"]
    return case["kappa"] * (1.0 + 0.05 * np.random.default_rng([5, seed]).uniform(-1, 1))


def _vectors(N, nrhs, cplx, seed):
    """Columns of normal entries, as the orthonormal vectors of a Krylov basis have them."""
    rng = np.random.default_rng([1, seed])
    x = rng.normal(size=(nrhs, N))
    return x + 1j * rng.normal(size=(nrhs, N)) if cplx else x


def _unit(rng, n):
    d = rng.normal(size=(n, 3))
    return d / np.linalg.norm(d, axis=1, keepdims=True)


def _data(case, seed):
    """(load-vector kind, its parameters, evaluation points): point sources outside the sphere, plane waves for
    Helmholtz, Hertz dipoles for Maxwell; 100 points inside the surface, for Maxwell of radius at most 0.25 too."""
    rng = np.random.default_rng([2, seed])
    k = case["nrhs"]
    if case["geometry"] == "torus":  # radii 2 and 0.5, axis z: points within 0.2 of the core circle
        ang, d = rng.uniform(0, 2 * np.pi, 100), _unit(rng, 100) * rng.uniform(0, 0.2, (100, 1))
        points = np.stack([2 * np.cos(ang), 2 * np.sin(ang), 0 * ang], 1) + d
        radius = rng.uniform(3.5, 5.0, (k, 1))
    else:
        points = _unit(rng, 100) * (0.25 * rng.uniform(0, 1, (100, 1)) ** (1 / 3))
        radius = rng.uniform(1.5, 3.0, (k, 1)) if case["operator"] == "laplace" else 2.5
    if case["operator"] == "laplace":
        return 0, _unit(rng, k) * radius, points
    if case["operator"] == "helmholtz":
        return 2, _unit(rng, k), points
    return 3, np.concatenate([_unit(rng, k) * radius, _unit(rng, k)], 1), points


def prepare(case, seed):
    op = _operator(case, _wavenumber(case, seed))
    state = {"case": case, "op": op, "A": op.get_discrete_operator()}
    if case["work"] != "assemble":
        op.compute()
    if case["work"] == "solve":
        state["kind"], state["params"], state["points"] = _data(case, seed)
    else:
        state["x"] = torch.from_numpy(_vectors(op.N, case["nrhs"], op.is_complex, seed)).cuda().t()
    return state


def run(state):
    case, op, A = state["case"], state["op"], state["A"]
    if case["work"] == "product":
        return A.matvec(state["x"], precision=case["precision"])
    if case["work"] == "assemble":
        op.compute()
        return A.matvec(state["x"])
    b = op.load_vector(state["kind"], state["params"])
    density, _ = A.solve(b, tol=SOLVE_TOL, inner=case["precision"])
    return op.potential(density, state["points"])


@functools.lru_cache(maxsize=64)
def _sizes(operator, geometry, M, P, n_p):
    """(unknowns, near-field entries, far-field couplings, integrand evaluations) from a host-only operator."""
    case = _case("product", operator, geometry, M, P, n_p, 1, "fp64", 1.0)
    op = _operator(case, 1.0, bg.Context(-1))
    info = op.info()
    near = op.n_dense * (int(info[5]) * int(info[11]) * (P + 1) ** 2) ** 2
    far = op.n_lowrank * n_p ** 4  # Maxwell's four component blocks come from the one kernel matrix
    evaluations = 0
    if operator != "maxwell":
        evaluations = sum(q["evaluations"] for q in op.quadrature_counts().values())
    return op.N, near, far, evaluations


def work(case):
    """Bytes: the operator's near-field entries and couplings read once (at the width the precision needs), x
    read, y written; an assembly writes them instead. Operations: a multiply-add per entry and column; an
    assembly's integrand evaluations at the 30 operations that points, distance, kernel and sum cannot do
    without. A solve is at least 50 products (unpreconditioned Krylov at these condition numbers)."""
    cplx = case["operator"] != "laplace"
    N, near, far, evaluations = _sizes(case["operator"], case["geometry"], case["M"], case["P"], case["n_p"])
    wide, k = (16 if cplx else 8), case["nrhs"]
    near_b = wide if case["precision"] != "fp32" else wide // 2
    far_b = wide if case["precision"] == "fp64" else wide // 2
    macs = near * k + far * k * (4 if case["operator"] == "maxwell" else 1)
    one = {"bytes": near * near_b + far * far_b + 2 * N * k * wide, "flops": macs * (8 if cplx else 2)}
    if case["work"] == "assemble":
        return {"bytes": (near + far) * wide, "flops": 30 * evaluations + one["flops"]}
    times = 50 if case["work"] == "solve" else 1
    return {"bytes": one["bytes"] * times, "flops": one["flops"] * times}


# ---- the same outputs in 64 bits, without the package ----

def _load_patches(geometry):
    """Homogeneous control nets (px, py, 4) of a .dat file of Bezier patches."""
    with open(os.path.join(GEO, geometry + ".dat")) as f:
        rows = [r.split() for r in f if not r.startswith("#")]
    count, rows, nets = int(rows[0][2]), rows[1:], []
    for p in range(count):
        block = rows[9 * p:9 * p + 9]
        px, py = int(block[2][0]), int(block[2][1])
        nets.append(np.array([[float(v) for v in r] for r in block[5:9]]).reshape(4, py, px).transpose(2, 1, 0))
    return np.array(nets)


def _bernstein(p, u):
    return torch.stack([math.comb(p, i) * u ** i * (1 - u) ** (p - i) for i in range(p + 1)], -1)


def _bernstein_d(p, u):
    b = _bernstein(p - 1, u)
    z = torch.zeros_like(b[..., :1])
    return p * (torch.cat([z, b], -1) - torch.cat([b, z], -1))


class _Surface:
    """Points and area elements of a patchwise mapped surface, and the elements of its refinement."""

    def __init__(self, geometry, M, P, device):
        self.device, self.P, self.n = device, P, 2 ** M
        self.nets = None if geometry == "cube" else torch.as_tensor(_load_patches(geometry), device=device)
        n = self.n
        e = torch.arange(PATCHES[geometry] * n * n, device=device)
        self.patch, self.i, self.j = e // (n * n), e % n, (e // n) % n
        self.dofs_per_side = n + P
        self.N = PATCHES[geometry] * self.dofs_per_side ** 2

    def frame(self, patch, s, t):
        """(points, area element) for patch (...) and coordinates s, t (..., q)."""
        if self.nets is None:  # x / |x| of the cube's faces
            k, pos = patch // 2, patch % 2 == 0
            a, b = (k + torch.where(pos, 1, 2)) % 3, (k + torch.where(pos, 2, 1)) % 3
            eye = torch.eye(3, dtype=torch.float64, device=self.device)
            ea, eb = 2 * eye[a][..., None, :], 2 * eye[b][..., None, :]
            c = (torch.where(pos, 1.0, -1.0).double()[..., None] * eye[k])[..., None, :] \
                + (s - 0.5)[..., None] * ea + (t - 0.5)[..., None] * eb
            r = c.norm(dim=-1, keepdim=True)
            x = c / r
            ds, dt = ((d - x * (x * d).sum(-1, keepdim=True)) / r for d in (ea, eb))
        else:
            px, py = self.nets.shape[1] - 1, self.nets.shape[2] - 1
            bs, bt = _bernstein(px, s), _bernstein(py, t)
            net = self.nets[patch]
            h, hs, ht = (torch.einsum("...qi,...qj,...ijc->...qc", u, v, net)
                         for u, v in ((bs, bt), (_bernstein_d(px, s), bt), (bs, _bernstein_d(py, t))))
            x, w = h[..., :3] / h[..., 3:], h[..., 3:]
            ds, dt = ((d[..., :3] - x * d[..., 3:]) / w for d in (hs, ht))
        return x, torch.linalg.cross(ds, dt).norm(dim=-1)

    def basis(self, e, u, v):
        """Values (..., q, (P+1)^2) and degrees of freedom (..., (P+1)^2) of the B-splines on elements e (...)
        at local coordinates u, v (..., q), times 2^M (the operator's scaling)."""
        P, side = self.P, self.dofs_per_side
        one = [self._splines(span[e], c) for span, c in ((self.i, u), (self.j, v))]
        values = (one[1][..., :, None] * one[0][..., None, :]).flatten(-2) * self.n
        k = torch.arange(P + 1, device=self.device)
        dof = (self.j[e][..., None, None] + k[:, None]) * side + self.i[e][..., None, None] + k
        return values, self.patch[e][..., None] * side * side + dof.flatten(-2)

    def _splines(self, span, u):
        """The P + 1 B-splines of open uniform knots (unit spacing) on a span, at span + u (Cox, de Boor)."""
        P, x = self.P, span[..., None] + u
        knot = lambda q: (span + q).clamp(0, self.n)[..., None].double()  # noqa: E731
        N = [torch.ones_like(u)]
        for d in range(1, P + 1):
            saved, new = torch.zeros_like(u), []
            for r in range(d):
                right, left = knot(r + 1), knot(r + 1 - d)
                part = N[r] / (right - left)
                new.append(saved + (right - x) * part)
                saved = (x - left) * part
            N = new + [saved]
        return torch.stack(N, -1)

    def at(self, e, u, v):
        """(points, area element) on elements e at local coordinates; the area element of the element's square."""
        x, g = self.frame(self.patch[e], (self.i[e][..., None] + u) / self.n, (self.j[e][..., None] + v) / self.n)
        return x, g / self.n ** 2


def _gauss(q, device):
    x, w = np.polynomial.legendre.leggauss(q)
    return torch.as_tensor((x + 1) / 2, device=device), torch.as_tensor(w / 2, device=device)


def _singular_rule(shared, q, device):
    """Points ((x1, x2), (y1, y2)) and weights on the unit square pair with the kernel's singularity at x = y
    (4 shared corners), at x1 = y1, x2 = y2 = 0 (2) or at the origin (1): relative coordinates and one pyramid
    per coordinate that may be the largest, whose apex variable cancels the singularity."""
    g, w = _gauss(q, device)
    r = torch.stack(torch.meshgrid(g, g, g, g, indexing="ij"), -1).reshape(-1, 4)
    wr = torch.einsum("a,b,c,d->abcd", w, w, w, w).reshape(-1)
    rules = []
    for top in range({4: 2, 2: 3, 1: 4}[shared]):
        dim = {4: 2, 2: 3, 1: 4}[shared]
        z = [r[:, 0] if k == top else r[:, 0] * r[:, 1 + (k if k < top else k - 1)] for k in range(dim)]
        jac = wr * r[:, 0] ** (dim - 1)
        if shared == 1:
            rules.append((z[0], z[1], z[2], z[3], jac))
        elif shared == 2:  # z = (|y1 - x1|, x2, y2); x1 over what is left of the edge
            low = (1 - z[0]) * r[:, 3]
            for a, b in ((low, low + z[0]), (low + z[0], low)):
                rules.append((a, z[1], b, z[2], jac * (1 - z[0])))
        else:  # z = |y - x| in both directions, four signs
            l1, l2 = (1 - z[0]) * r[:, 2], (1 - z[1]) * r[:, 3]
            for a1, b1 in ((l1, l1 + z[0]), (l1 + z[0], l1)):
                for a2, b2 in ((l2, l2 + z[1]), (l2 + z[1], l2)):
                    rules.append((a1, a2, b1, b2, jac * (1 - z[0]) * (1 - z[1])))
    return [torch.cat(c) for c in zip(*rules)]


_CORNERS = ((0, 0), (1, 0), (1, 1), (0, 1))


def _oriented(first, second, u, v, device):
    """Local coordinates of (u, v) when u runs from corner first to corner second and v away from that side."""
    c = torch.tensor(_CORNERS, dtype=torch.float64, device=device)
    a, along = c[first], c[second] - c[first]
    inward = torch.where(along == 0, 1 - 2 * a, torch.zeros_like(a))
    return [a[:, d, None] + along[:, d, None] * u + inward[:, d, None] * v for d in (0, 1)]


def _kernel(r, kappa):
    k = 1 / (4 * math.pi * r)
    return k * torch.exp(-1j * kappa * r) if kappa else k


def _galerkin_product(case, kappa, x):
    """y = A x of the Galerkin matrix itself (x (N, k)): Gauss rules for pairs of elements that do not touch,
    the rules above for those that do."""
    dev = x.device
    S = _Surface(case["geometry"], case["M"], case["P"], dev)
    ne = S.patch.numel()
    e = torch.arange(ne, device=dev)
    y = torch.zeros_like(x)

    corner = torch.tensor(_CORNERS, dtype=torch.float64, device=dev)
    pts = S.at(e, corner[:, 0].expand(ne, 4), corner[:, 1].expand(ne, 4))[0].reshape(-1, 3)
    _, vertex = torch.unique((pts * 1e6).round().long(), dim=0, return_inverse=True)
    vertex = vertex.reshape(ne, 4)
    same = vertex[:, None, :, None] == vertex[None, :, None, :]  # (ne, ne, 4, 4)
    shared = same.any(-1).sum(-1)

    q = 6
    g, w = _gauss(q, dev)
    u, v = (c.reshape(-1).expand(ne, q * q) for c in torch.meshgrid(g, g, indexing="ij"))
    X, area = S.at(e, u, v)
    phi, dof = S.basis(e, u, v)
    phi = phi * (area * (w[:, None] * w[None, :]).reshape(-1))[..., None]
    rho = torch.einsum("eqb,ebk->eqk", phi.to(x.dtype), x[dof]).reshape(ne * q * q, -1)
    flat, step = X.reshape(-1, 3), max(1, (1 << 24) // (ne * q ** 4))
    for a in range(0, ne, step):
        b = min(ne, a + step)
        r = (flat[a * q * q:b * q * q, None] - flat[None]).norm(dim=-1).reshape(b - a, q * q, ne, q * q)
        far = (shared[a:b] == 0)[:, None, :, None]
        K = _kernel(torch.where(far, r, torch.ones_like(r)), kappa) * far
        pot = (K.reshape((b - a) * q * q, -1) @ rho).reshape(b - a, q * q, -1)
        y.index_put_((dof[a:b],), torch.einsum("eqb,eqk->ebk", phi[a:b].to(x.dtype), pot), accumulate=True)

    for kind in (4, 2, 1):
        x1, x2, y1, y2, wt = _singular_rule(kind, 7, dev)
        left, right = torch.nonzero(shared == kind, as_tuple=True)
        step = max(1, (1 << 20) // wt.numel())
        for a in range(0, left.numel(), step):
            la, rb = left[a:a + step], right[a:a + step]
            m = same[la, rb].to(torch.int8)
            if kind == 4:
                sides = [torch.zeros_like(la), torch.ones_like(la)] * 2
            else:  # corners of the left element that the right one has, and theirs there
                has = m.amax(-1)
                first = has.argmax(-1)
                second = 3 - has.flip(-1).argmax(-1) if kind == 2 else (first + 1) % 4
                other = [m[torch.arange(la.numel(), device=dev), c].argmax(-1) for c in (first, second)]
                sides = [first, second, other[0], other[1] if kind == 2 else (other[0] + 1) % 4]
            ua, va = _oriented(sides[0], sides[1], x1, x2, dev)
            ub, vb = _oriented(sides[2], sides[3], y1, y2, dev)
            (Xa, ga), (Xb, gb) = S.at(la, ua, va), S.at(rb, ub, vb)
            (fa, da), (fb, db) = S.basis(la, ua, va), S.basis(rb, ub, vb)
            c = _kernel((Xa - Xb).norm(dim=-1), kappa) * ga * gb * wt
            block = torch.einsum("pqa,pqb->pab", fa.to(c.dtype) * c[..., None], fb.to(c.dtype))
            y.index_put_((da,), torch.einsum("pab,pbk->pak", block, x[db]), accumulate=True)
    return y


def exact(case, seed):
    """Solves: the analytic field of the data at the points. Products and assemblies of the scalar operators up
    to MAX_EXACT_ELEMENTS elements: the Galerkin matrix by direct quadrature (the H2 matrix differs from it by
    its interpolation). Others: none (Maxwell's dense matrix, larger products: too long)."""
    kappa = _wavenumber(case, seed)
    if case["work"] == "solve":
        kind, prm, pts = _data(case, seed)
        if kind == 2:
            return np.exp(-1j * kappa * (pts @ prm.T))
        c = pts[:, None, :] - prm[None, :, :3]
        r = np.linalg.norm(c, axis=2, keepdims=True)
        if kind == 0:
            return 1 / (4 * np.pi * r[..., 0])
        n, mom = c / r, np.broadcast_to(prm[None, :, 3:], c.shape)
        wave = np.exp(-1j * kappa * r)
        along = (n * mom).sum(2, keepdims=True) * n
        field = kappa ** 2 * wave / r * (mom - along) + (1 / r ** 3 + 1j * kappa / r ** 2) * wave * (3 * along - mom)
        return field.transpose(0, 2, 1)
    elements = PATCHES[case["geometry"]] * 4 ** case["M"]
    if case["operator"] == "maxwell" or elements > MAX_EXACT_ELEMENTS:
        return None
    N = PATCHES[case["geometry"]] * (2 ** case["M"] + case["P"]) ** 2
    x = torch.from_numpy(_vectors(N, case["nrhs"], case["operator"] != "laplace", seed))
    x = x.cuda() if torch.cuda.is_available() else x
    return _galerkin_product(case, kappa, x.t().contiguous())
