"""Performance cases: the calls a user of this package makes, over the sizes it makes them at.

Families (one public call, or one pair of calls that belong together, per case):

  maps      eval and grad of a nodal field at the quadrature points and their reverse mode:
            what a user-written energy ``op.integrate(psi(op.eval(u), op.grad(u)))`` costs
            besides psi, forward and backward
  energy    energy and residual at one state: what a line search or an explicit step evaluates
  hvp       matrix-free Hessian-vector product: one Krylov iteration's operator
  assemble  residual and sparse tangent in one call: one Newton iteration's assembly
  solve     a clamped structured brick under traction, to relative residual 1e-10
  batch     many independent Poisson problems of uneven size in one launch
  serve     a backlog of brick solves of mixed sizes through the request loop

Meshes, plans, colourings and resident models do not depend on the inputs' seed: a program
builds them once and keeps them, and so does ``prepare`` (a bounded cache).
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from tatva_gb300 import Mesh, Operator, batched, element, materials, problems, serving, solvers, sparse

DEV = "cuda"
DTYPES = {"f32": torch.float32, "f64": torch.float64}


# ------------------------------------------------------------------------------- cases
def listed():
    return [
        # 2D Poisson on the unit square, 8192 triangles: the smallest assembly in use
        dict(name="assemble_tri3_poisson_64", family="assemble", element="tri3", law="poisson",
             nx=64, ny=64, nz=0, jitter=0.0, dtype="f64"),
        # Newton tangent of a hyperelastic block (Kuhn tets, jittered), FP32 as in Newton
        dict(name="assemble_tet4_neohooke_56", family="assemble", element="tet4",
             law="neohooke", nx=56, ny=56, nz=56, jitter=0.2, dtype="f32"),
        # user-written energies on tets: vector field, FP64, forward and backward
        dict(name="maps_tet4_f64_44", family="maps", element="tet4", nx=44, ny=44, nz=44,
             jitter=0.2, dtype="f64", vals=3),
        # ... on a regular brick in FP32
        dict(name="maps_hex8_f32_96x80x112", family="maps", element="hex8", nx=96, ny=80, nz=112,
             jitter=0.0, dtype="f32", vals=3),
        # ... a scalar field (temperature, phase field) on a distorted hex mesh of odd size
        dict(name="maps_hex8_f64_61x67x59", family="maps", element="hex8", nx=61, ny=67, nz=59,
             jitter=0.2, dtype="f64", vals=1),
        # Newton's FP64 residual with its line-search energy on a distorted hex mesh
        dict(name="energy_hex8_neohooke_f64", family="energy", element="hex8", law="neohooke",
             nx=48, ny=40, nz=44, jitter=0.2, dtype="f64"),
        # the Hex8 elasticity operator of the 128^3 brick solve
        dict(name="hvp_hex8_brick_f32_128", family="hvp", element="hex8", law="elastic", nx=128,
             ny=128, nz=128, jitter=0.0, dtype="f32", fixed=True),
        # the same law on a distorted mesh of odd size
        dict(name="hvp_hex8_jitter_f32", family="hvp", element="hex8", law="elastic", nx=96,
             ny=90, nz=101, jitter=0.2, dtype="f32", fixed=True),
        # matrix-free operator of the 5.3 M tet hyperelastic block
        dict(name="hvp_tet4_neohooke_f32_96", family="hvp", element="tet4", law="neohooke",
             nx=96, ny=96, nz=96, jitter=0.2, dtype="f32", fixed=True),
        # one mixed-precision solve of the largest served brick
        dict(name="solve_brick_mixed_64", family="solve", nx=64, ny=64, nz=64, method="mixed"),
        # unit squares of side 8..96, lognormal conductivity, in one launch
        dict(name="batch_poisson_768", family="batch", count=768, side_min=8, side_max=96),
        # requests of sides 16..64 through the continuous-batching loop
        dict(name="serve_mix_24", family="serve", count=24, side_max=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng, elem, lo, hi):
    """Cells along each axis: a log-uniform size, each axis up to 30 % off it."""
    n = _log_int(rng, lo, hi)
    d = [max(2, min(hi, int(round(n * rng.uniform(0.75, 1.3))))) for _ in range(3)]
    return dict(nx=d[0], ny=d[1], nz=0 if elem == "tri3" else d[2])


def draw(rng):
    fam = rng.choice(["maps", "maps", "maps", "energy", "hvp", "hvp", "hvp", "assemble",
                      "assemble", "solve", "batch", "serve"])
    if fam == "solve":
        return dict(family=fam, **_dims(rng, "hex8", 12, 64),
                    method=rng.choice(["mixed", "mixed", "fp64"]))
    if fam == "batch":
        lo = _log_int(rng, 6, 24)
        return dict(family=fam, count=_log_int(rng, 48, 700), side_min=lo,
                    side_max=max(lo + 1, _log_int(rng, 24, 96)))
    if fam == "serve":
        return dict(family=fam, count=rng.randrange(4, 25), side_max=rng.choice([24, 32, 48, 64]))
    elem = rng.choice(["tri3", "tet4", "tet4", "hex8", "hex8"])
    top = {"maps": dict(tri3=900, tet4=48, hex8=88), "energy": dict(tri3=900, tet4=72, hex8=48),
           "hvp": dict(tri3=1024, tet4=84, hex8=100),
           "assemble": dict(tri3=512, tet4=44, hex8=36)}[fam][elem]
    low = dict(tri3=12, tet4=6, hex8=6)[elem]
    c = dict(family=fam, element=elem, **_dims(rng, elem, low, top),
             jitter=rng.choice([0.0, 0.2]), dtype=rng.choice(["f32", "f64"]))
    if fam == "maps":
        return dict(c, vals=rng.choice([1, 1, 2, 3, 3, 6]))
    c["law"] = rng.choice(["poisson", "elastic"] + ([] if elem == "tri3" else ["neohooke"]))
    if fam == "hvp":
        c["fixed"] = rng.random() < 0.7
    return c


# -------------------------------------------------------------------------------- meshes
def _mesh_arrays(element_, nx, ny, nz, jitter):
    """Coordinates and connectivity of the unit square (triangles) or unit cube (hexahedra;
    six tetrahedra per cell), interior nodes moved by up to jitter cells along each axis."""
    n = [nx, ny] if element_ == "tri3" else [nx, ny, nz]
    axes = [np.linspace(0.0, 1.0, k + 1) for k in n]
    if element_ == "tri3":
        c = np.stack([a.ravel() for a in np.meshgrid(*axes, indexing="ij")], -1)
        i, j = (a.ravel() for a in np.meshgrid(np.arange(nx), np.arange(ny), indexing="ij"))
        p = i * (ny + 1) + j
        q = p + ny + 1
        el = np.stack([np.stack([p, q, q + 1], 1), np.stack([p, q + 1, p + 1], 1)], 1)
        el = el.reshape(-1, 3)
    else:
        z, y, x = np.meshgrid(axes[2], axes[1], axes[0], indexing="ij")
        c = np.stack([x.ravel(), y.ravel(), z.ravel()], -1)
        k, j, i = (a.ravel() for a in np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx),
                                                  indexing="ij"))
        sy, sz = nx + 1, (nx + 1) * (ny + 1)
        p = i + j * sy + k * sz
        v = [p, p + 1, p + sy, p + sy + 1, p + sz, p + sz + 1, p + sz + sy, p + sz + sy + 1]
        if element_ == "hex8":
            el = np.stack([v[a] for a in (0, 1, 3, 2, 4, 5, 7, 6)], 1)
        else:
            t = ((0, 1, 3, 7), (0, 1, 7, 5), (0, 5, 7, 4), (0, 3, 2, 7), (0, 2, 6, 7), (0, 6, 4, 7))
            el = np.stack([np.stack([v[a] for a in r], -1) for r in t], 1).reshape(-1, 4)
    if jitter:
        inside = np.all((c > 1e-12) & (c < 1 - 1e-12), axis=1)
        d = np.random.default_rng(3).uniform(-jitter, jitter, size=c.shape) / np.array(n)
        c[inside] += d[inside]
    return c, el.astype(np.int32)


ELEMENTS = {"tri3": element.Tri3, "tet4": element.Tetrahedron4, "hex8": element.Hexahedron8}
LAWS = {  # parameters of each law
    "poisson": (1.3, 0.7),
    "elastic": (1 / 2.6, 0.3 / (0.4 * 1.3)),
    "neohooke": (1.0, 10.0),
}


@functools.lru_cache(maxsize=2)
def _model(elem, nx, ny, nz, jitter, law, want_plan, want_matrix):
    """What a program builds once per mesh and keeps."""
    c, el = _mesh_arrays(elem, nx, ny, nz, jitter)
    op = Operator(Mesh(c, el, device=DEV), ELEMENTS[elem]())
    en = None
    if law:
        kind = dict(poisson=materials.Poisson, elastic=materials.LinearElastic,
                    neohooke=materials.NeoHookean)[law]
        en = kind(op, *LAWS[law])
    if want_plan:
        en.plan()
    else:
        op.incidence()
    jac = None
    if want_matrix:
        cm = sparse.ColoredMatrix.from_csr(sparse.pattern_from_mesh(op.mesh, en.n_values),
                                           device=DEV)
        jac = sparse.linearized_jacfwd(en.residual, cm)
    return op, en, jac


def _op_of(case):
    fam = case["family"]
    return _model(case["element"], case["nx"], case["ny"], case["nz"], case["jitter"],
                  case.get("law", ""), fam != "maps", fam == "assemble")


@functools.lru_cache(maxsize=2)
def _brick(nx, ny, nz):
    """Clamped brick [0,1]^3 of nx x ny x nz cells and its unit face load."""
    if nx == ny == nz:
        P = problems.clamped_brick(nx, DEV, traction=1.0)
        P["energy"].plan()
        return P["energy"], P["fixed"], P["b"]
    c, el = _mesh_arrays("hex8", nx, ny, nz, 0.0)
    op = Operator(Mesh(c, el, device=DEV), element.Hexahedron8())
    en = materials.LinearElastic.from_young(op, 1.0, 0.3)
    en.plan()
    fixed, load = _clamp(c, nx, ny, nz)
    return en, fixed, load


def _clamp(c, nx, ny, nz):
    left, right = c[:, 0] == 0.0, np.where(c[:, 0] == 1.0)[0]
    fixed = torch.from_numpy(np.repeat(left, 3).astype(np.uint8)).to(DEV)
    edge = [np.isclose(c[right, d], 0.0) | np.isclose(c[right, d], 1.0) for d in (1, 2)]
    load = np.zeros(c.size)
    load[right * 3] = np.where(edge[0], 1, 2) * np.where(edge[1], 1, 2) / (4.0 * ny * nz)
    return fixed, torch.from_numpy(load).to(DEV)


@functools.lru_cache(maxsize=1)
def _batch(count, lo, hi):
    meshes, kappas, _ = batched.random_unit_squares(count, lo, hi, seed=11)
    systems, b, _ = batched.poisson_batch(meshes, kappas, f=1.0, device=DEV)
    return systems, b, meshes, kappas


@functools.lru_cache(maxsize=1)
def _server(side_max):
    srv = serving.Server(DEV, slots=64, keep_solutions=True)
    srv.warm(_sides(side_max))
    return srv


def _sides(side_max):
    return tuple(s for s in (16, 24, 32, 48, 64) if s <= side_max)


# -------------------------------------------------------------------------------- inputs
def _field(c, vals, gen, amp, noise):
    """A smooth nodal field (three waves per component) with node-to-node noise."""
    d = c.shape[1]
    out = torch.zeros(c.shape[0], vals, dtype=torch.float64, device=DEV)
    for _ in range(3):
        k = (torch.rand(d, vals, generator=gen, device=DEV, dtype=torch.float64) - 0.5) * 10
        ph = torch.rand(vals, generator=gen, device=DEV, dtype=torch.float64) * 6.3
        out += torch.sin(c @ k + ph)
    rough = torch.randn(out.shape, generator=gen, device=DEV, dtype=torch.float64)
    return amp * out + noise * rough


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _vectors(case, coords, seed, n_quad=0, n_elems=0):
    """The nodal inputs of one pass (the same for prepare and exact)."""
    g, dt, fam = _gen(seed), DTYPES[case["dtype"]], case["family"]
    h = 1.0 / max(case["nx"], case["ny"], case["nz"])
    dim = coords.shape[1]
    if fam == "maps":
        V = case["vals"]
        u = _field(coords, V, g, 0.5, 0.05).to(dt)
        cq = torch.randn(n_elems, n_quad, V, generator=g, device=DEV, dtype=dt)
        cg = torch.randn(n_elems, n_quad, V, dim, generator=g, device=DEV, dtype=dt)
        if V == 1:  # a scalar field has no component axis
            u, cq, cg = u[:, 0].contiguous(), cq[..., 0].contiguous(), cg[:, :, 0].contiguous()
        return dict(u=u, cq=cq, cg=cg)
    V = 1 if case["law"] == "poisson" else dim
    s = dict(u=_field(coords, V, g, 0.01, 0.01 * h).to(dt).reshape(-1))
    if fam == "hvp":
        s["v"] = _field(coords, V, g, 0.3, 0.1).to(dt).reshape(-1)
        s["fixed"] = None
        if case["fixed"]:  # held face x = 0, where a Krylov direction is zero
            s["fixed"] = (coords[:, :1] < 1e-12).expand(-1, V).to(torch.uint8).reshape(-1)
            s["v"] = torch.where(s["fixed"].bool(), 0.0, s["v"])
    return s


def _solve_load(case, load, seed):
    t = torch.randn(3, generator=_gen(seed), device=DEV, dtype=torch.float64) * 1e-3
    return (load.view(-1, 3)[:, :1] * t).reshape(-1).contiguous()


def _batch_load(b, seed):
    i = torch.arange(b.numel(), device=DEV, dtype=torch.float64)
    p = torch.rand(2, generator=_gen(seed), device=DEV, dtype=torch.float64)
    return b * (1.0 + 0.5 * torch.sin(i * (0.002 + 0.01 * p[0]) + 6.3 * p[1]))


def _requests(case, seed):
    """A backlog: every side in turn (the case's), material and load from the seed."""
    rng, sides = np.random.default_rng(int(seed) & 0x7FFFFFFF), _sides(case["side_max"])
    return [serving.SolveRequest(i, 0.0, sides[(7 * i + 3) % len(sides)],
                                 float(rng.lognormal(0.0, 0.5)), float(rng.uniform(0.2, 0.45)),
                                 float(rng.uniform(0.5, 1.5)) * 1e-3)
            for i in range(case["count"])]


def prepare(case, seed):
    fam = case["family"]
    if fam == "solve":
        en, fixed, load = _brick(case["nx"], case["ny"], case["nz"])
        return dict(family=fam, method=case["method"], energy=en, fixed=fixed,
                    b=_solve_load(case, load, seed))
    if fam == "batch":
        systems, b, _, _ = _batch(case["count"], case["side_min"], case["side_max"])
        return dict(family=fam, systems=systems, b=_batch_load(b, seed))
    if fam == "serve":
        return dict(family=fam, server=_server(case["side_max"]), requests=_requests(case, seed))
    op, en, jac = _op_of(case)
    s = _vectors(case, op.mesh.coords, seed, op.n_quad, op.n_elements)
    if fam == "maps":
        s["u"].requires_grad_(True)
    return dict(s, family=fam, op=op, energy=en, jac=jac, linear=case.get("law") != "neohooke")


def run(s):
    fam = s["family"]
    if fam == "maps":
        q, g = s["op"].eval(s["u"]), s["op"].grad(s["u"])
        (du,) = torch.autograd.grad((q, g), s["u"], (s["cq"], s["cg"]))
        return dict(q=q.detach(), g=g.detach(), du=du)
    if fam == "energy":
        return dict(value=s["energy"].value(s["u"]), residual=s["energy"].residual(s["u"]))
    if fam == "hvp":
        return s["energy"].hvp(None if s["linear"] else s["u"], s["v"], fixed=s["fixed"])
    if fam == "assemble":
        r, K = s["jac"](s["u"])
        return dict(residual=r, data=K.data)
    if fam == "solve":
        solver = solvers.mixed_cg if s["method"] == "mixed" else solvers.cg
        return solver(s["energy"], s["b"], fixed=s["fixed"], rtol=1e-10).x
    if fam == "batch":
        return s["systems"].solve(s["b"]).x
    return [r.x for r in s["server"].run(s["requests"], realtime=False).records]


# ---------------------------------------------------------------------------------- work
def _counts(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case.get("element") == "tri3":
        return (nx + 1) * (ny + 1), 2 * nx * ny, 3, 2, 1
    nn = (nx + 1) * (ny + 1) * (nz + 1)
    return (nn, 6 * nx * ny * nz, 4, 3, 1) if case.get("element") == "tet4" else \
        (nn, nx * ny * nz, 8, 3, 8)


def _element_flops(npe, dim, quad, V):
    """Geometry (Jacobian, inverse), gradient, law and its transpose, per quadrature point."""
    return quad * (2 * npe * dim * (dim + 2 * V) + 40 + 6 * V * dim * dim)


def work(case):
    fam = case["family"]
    if fam == "batch":  # the matrix once, b and x; CG iterations grow with the side
        lo, hi = case["side_min"], case["side_max"]
        p = lambda k: (hi ** k - lo ** k) / (k * math.log(hi / lo))  # noqa: E731
        rows = case["count"] * p(2)
        return dict(bytes=rows * (7 * 12 + 16), flops=case["count"] * p(3) * 3.5 * 24)
    if fam == "serve":
        n = _sides(case["side_max"])
        per = sum((s + 1) ** 3 * 3 for s in n) / len(n)
        return dict(bytes=case["count"] * per * 16, flops=case["count"] * sum(
            (s + 1) ** 3 * 200.0 * 16 * s for s in n) / len(n))
    nn, E, npe, dim, quad = _counts(dict(case, element=case.get("element", "hex8")))
    if fam == "solve":
        return dict(bytes=nn * 3 * 16 + nn * 3,
                    flops=nn * 200.0 * 9 * max(case["nx"], case["ny"], case["nz"]))
    sz = 4 if case["dtype"] == "f32" else 8
    V = case["vals"] if fam == "maps" else (1 if case["law"] == "poisson" else dim)
    mesh = 4 * npe * E + sz * dim * nn
    fl = E * _element_flops(npe, dim, quad, V)
    if fam == "maps":
        return dict(bytes=mesh + sz * (2 * nn * V + 2 * E * quad * V * (1 + dim)), flops=2 * fl)
    if fam == "energy":
        return dict(bytes=mesh + sz * 2 * nn * V, flops=2 * fl)
    if fam == "hvp":
        vecs = 3 if case["law"] == "neohooke" else 2
        if case["jitter"] == 0.0 and case["element"] == "hex8" and case["law"] == "elastic":
            mesh = 0  # a uniform brick's operator needs no mesh data
        return dict(bytes=mesh + sz * vecs * nn * V + (nn * V if case["fixed"] else 0), flops=fl)
    pairs = {"tri3": 7, "tet4": 15, "hex8": 27}[case["element"]]  # neighbours per node
    return dict(bytes=mesh + sz * (2 * nn * V + nn * pairs * V * V),
                flops=fl + E * quad * (npe * V) ** 2 * 2 * dim)


# --------------------------------------------------------------------------------- exact
def _reference_points(elem):
    """(weights (Q,), N (Q, A), dN (Q, A, D)) of the reference element."""
    if elem != "hex8":
        d = 2 if elem == "tri3" else 3
        dN = np.concatenate([-np.ones((1, d)), np.eye(d)])[None]
        N = np.full((1, d + 1), 1.0 / (d + 1))
        return np.array([0.5 if d == 2 else 1 / 6]), N, dN
    s = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1],
                  [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]], float)
    x = s / math.sqrt(3.0)
    f = 1 + s[None] * x[:, None]  # (Q, A, 3)
    N = f.prod(-1) / 8
    dN = np.stack([s[None, :, d] * np.delete(f, d, 2).prod(-1) for d in range(3)], -1) / 8
    return np.ones(8), N, dN


def _geometry(elem, X):
    """G (e, q, a, d) = dN_a/dx_d and the weights (e, q) for corner coordinates X (e, a, d)."""
    w, _, dN = (torch.as_tensor(t, dtype=torch.float64, device=DEV) for t in _reference_points(elem))
    J = torch.einsum("qai,eaj->eqij", dN, X)  # dx_j / dxi_i
    return torch.einsum("eqki,qai->eqak", torch.linalg.inv(J), dN), torch.linalg.det(J) * w


def _stress(law, H):
    p0, p1 = LAWS[law]
    if law == "poisson":
        return p0 * H
    if law == "elastic":
        tr = H.diagonal(dim1=-2, dim2=-1).sum(-1)[..., None, None]
        return p0 * (H + H.mT) + p1 * tr * torch.eye(H.shape[-1], dtype=H.dtype, device=DEV)
    F = H + torch.eye(3, dtype=H.dtype, device=DEV)
    Fit = torch.linalg.inv(F).mT
    lnJ = torch.log(torch.linalg.det(F))[..., None, None]
    return p0 * (F - Fit) + p1 * lnJ * Fit


def _moduli(law, H, dim):
    """A[..., i, J, k, L] = dP_iJ / dH_kL."""
    p0, p1 = LAWS[law]
    I = torch.eye(dim, dtype=torch.float64, device=DEV)
    if law == "poisson":
        return (p0 * I)[None, None, None, :, None, :].expand(H.shape[0], H.shape[1], 1, dim, 1, dim)
    if law == "elastic":
        A = p0 * (torch.einsum("ik,jl->ijkl", I, I) + torch.einsum("il,jk->ijkl", I, I)) \
            + p1 * torch.einsum("ij,kl->ijkl", I, I)
        return A.expand(H.shape[:2] + A.shape)
    F = H + I
    Fi = torch.linalg.inv(F)
    lnJ = torch.log(torch.linalg.det(F))[..., None, None, None, None]
    return (p0 * torch.einsum("ik,jl->ijkl", I, I)
            + (p0 - p1 * lnJ) * torch.einsum("eqjk,eqli->eqijkl", Fi, Fi)
            + p1 * torch.einsum("eqji,eqlk->eqijkl", Fi, Fi))


def _density(law, H, uq):
    p0, p1 = LAWS[law]
    if law == "poisson":
        return 0.5 * p0 * (H * H).sum((-1, -2)) - p1 * uq[..., 0]
    if law == "elastic":
        eps = 0.5 * (H + H.mT)
        return p0 * (eps * eps).sum((-1, -2)) + 0.5 * p1 * H.diagonal(dim1=-2, dim2=-1).sum(-1) ** 2
    F = H + torch.eye(3, dtype=H.dtype, device=DEV)
    lnJ = torch.log(torch.linalg.det(F))
    return 0.5 * p0 * ((F * F).sum((-1, -2)) - 3 - 2 * lnJ) + 0.5 * p1 * lnJ ** 2


def _cells(el, size=60000):
    return (el[k:k + size] for k in range(0, el.shape[0], size))


def _exact_mesh(case):
    c, el = _mesh_arrays(case["element"], case["nx"], case["ny"], case["nz"], case["jitter"])
    return torch.from_numpy(c).to(DEV), torch.from_numpy(el).to(DEV).long()


def _exact_maps(case, seed):
    c, el = _exact_mesh(case)
    _, N, _ = (torch.as_tensor(t, dtype=torch.float64, device=DEV)
               for t in _reference_points(case["element"]))
    s = {k: t.double() for k, t in _vectors(case, c, seed, N.shape[0], el.shape[0]).items()}
    if case["vals"] == 1:
        s = dict(u=s["u"][:, None], cq=s["cq"][..., None], cg=s["cg"][:, :, None])
    du = torch.zeros_like(s["u"])
    q, g, at = [], [], 0
    for e in _cells(el):
        G, _ = _geometry(case["element"], c[e])
        cq, cg = s["cq"][at:at + len(e)], s["cg"][at:at + len(e)]
        at += len(e)
        q.append(torch.einsum("qa,eav->eqv", N, s["u"][e]))
        g.append(torch.einsum("eqad,eav->eqvd", G, s["u"][e]))
        y = torch.einsum("qa,eqv->eav", N, cq) + torch.einsum("eqad,eqvd->eav", G, cg)
        du.index_add_(0, e.reshape(-1), y.reshape(-1, du.shape[1]))
    q, g = torch.cat(q), torch.cat(g)
    if case["vals"] == 1:
        q, g, du = q[..., 0], g[:, :, 0], du[:, 0]
    return dict(q=q, g=g, du=du)


def _exact_state(case, seed, want):
    """energy value / residual / hvp / CSR data at the case's inputs."""
    law, elem = case["law"], case["element"]
    c, el = _exact_mesh(case)
    _, N, _ = (torch.as_tensor(t, dtype=torch.float64, device=DEV) for t in _reference_points(elem))
    s = _vectors(case, c, seed)
    dim, nn = c.shape[1], c.shape[0]
    V = 1 if law == "poisson" else dim
    u = s["u"].double().view(nn, V)
    out = {}
    if "residual" in want:
        out["residual"] = torch.zeros(nn, V, dtype=torch.float64, device=DEV)
    if "value" in want:
        out["value"] = torch.zeros((), dtype=torch.float64, device=DEV)
    if "hvp" in want:
        fx = s["fixed"].view(nn, V).bool() if s["fixed"] is not None else None
        v0 = s["v"].double().view(nn, V)
        v = v0 if fx is None else torch.where(fx, 0.0, v0)
        out["hvp"] = torch.zeros(nn, V, dtype=torch.float64, device=DEV)
    if "data" in want:  # sorted (row, column) keys of the pattern, built per node pair
        A = el.shape[1]
        pairs = torch.cat([torch.unique((e[:, :, None] * nn + e[:, None, :]).reshape(-1))
                           for e in _cells(el, 2_000_000)])
        pairs = torch.unique(pairs)
        row, col = pairs // nn, pairs % nn
        blocks = torch.zeros(pairs.numel(), V, V, dtype=torch.float64, device=DEV)
    for e in _cells(el):
        G, w = _geometry(elem, c[e])
        H = torch.einsum("eqad,eav->eqvd", G, u[e])
        if "value" in want:
            out["value"] += (w * _density(law, H, torch.einsum("qa,eav->eqv", N, u[e]))).sum()
        if "residual" in want:
            y = torch.einsum("eqvd,eqad,eq->eav", _stress(law, H), G, w)
            if law == "poisson":
                y -= LAWS[law][1] * torch.einsum("qa,eq->ea", N, w)[..., None]
            out["residual"].index_add_(0, e.reshape(-1), y.reshape(-1, V))
        if "hvp" in want:
            dH = torch.einsum("eqad,eav->eqvd", G, v[e])
            dP = torch.einsum("eqijkl,eqkl->eqij", _moduli(law, H, dim), dH)
            y = torch.einsum("eqvd,eqad,eq->eav", dP, G, w)
            out["hvp"].index_add_(0, e.reshape(-1), y.reshape(-1, V))
        if "data" in want:
            AG = torch.einsum("eqijkl,eqbl,eq->eqijbk", _moduli(law, H, dim), G, w)
            K = torch.einsum("eqaj,eqijbk->eabik", G, AG)
            at = torch.searchsorted(pairs, (e[:, :, None] * nn + e[:, None, :]).reshape(-1))
            blocks.index_add_(0, at, K.reshape(-1, V, V))
    if "hvp" in want and fx is not None:
        out["hvp"] = torch.where(fx, v0, out["hvp"])
    for k in ("residual", "hvp"):
        if k in out:
            out[k] = out[k].reshape(-1)
    if "data" in want:
        # block (row, col) k-th of its row: entry (i, j) sits at V V start + i V len + k V + j
        per = torch.bincount(row, minlength=nn)
        start = torch.cumsum(per, 0) - per
        k = torch.arange(pairs.numel(), device=DEV) - start[row]
        i = torch.arange(V, device=DEV)
        at = (V * V * start[row])[:, None, None] + (i[:, None] * V * per[row][:, None, None]) \
            + (k * V)[:, None, None] + i[None, None, :]
        data = torch.empty(blocks.numel(), dtype=torch.float64, device=DEV)
        data[at.reshape(-1)] = blocks.reshape(-1)
        out["data"] = data
    return out["hvp"] if want == ("hvp",) else out


def _pcg(apply, b, dinv, tol, group=None, n_group=1, maxiter=6000):
    """Jacobi-CG in 64 bits, scalars per group of rows (independent systems)."""
    def dot(x, y):
        if group is None:
            return torch.dot(x, y)[None]
        return torch.zeros(n_group, dtype=torch.float64, device=DEV).index_add_(0, group, x * y)

    def per_row(s):
        return s[group] if group is not None else s
    x, r = torch.zeros_like(b), b.clone()
    z = r * dinv
    p, rz, b2 = z.clone(), dot(r, z), dot(b, b)
    for it in range(maxiter):
        q = apply(p)
        a = torch.nan_to_num(rz / dot(p, q), 0.0, 0.0, 0.0)
        x += per_row(a) * p
        r -= per_row(a) * q
        if it % 20 == 19 and bool((dot(r, r) <= tol * tol * b2).all()):
            break
        z = r * dinv
        new = dot(r, z)
        p = z + per_row(torch.nan_to_num(new / rz, 0.0, 0.0, 0.0)) * p
        rz = new
    return x


def _exact_brick(nx, ny, nz, mu, lam, b, fixed):
    """K x = b of the clamped brick: one element matrix for every cell."""
    _, el = _mesh_arrays("hex8", nx, ny, nz, 0.0)
    e = torch.from_numpy(el).to(DEV).long()
    X = torch.from_numpy(np.array([[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0], [0, 0, 1],
                                   [1, 0, 1], [1, 1, 1], [0, 1, 1]], float)
                         / np.array([nx, ny, nz], float)).to(DEV)
    G, w = _geometry("hex8", X[None])
    I = torch.eye(3, dtype=torch.float64, device=DEV)
    A = mu * (torch.einsum("ik,jl->ijkl", I, I) + torch.einsum("il,jk->ijkl", I, I)) \
        + lam * torch.einsum("ij,kl->ijkl", I, I)
    Ke = torch.einsum("eqaj,ijkl,eqbl,eq->aibk", G, A, G, w).reshape(24, 24)
    free = 1.0 - fixed.double()
    dofs = (e[:, :, None] * 3 + torch.arange(3, device=DEV)).reshape(-1)

    def apply(x):
        y = torch.zeros_like(x)
        y.index_add_(0, dofs, ((x * free)[dofs].view(-1, 24) @ Ke).reshape(-1))
        return y * free + x * (1 - free)

    d = torch.zeros_like(b)
    d.index_add_(0, dofs, Ke.diagonal().repeat(e.shape[0]))
    return _pcg(apply, b, 1.0 / torch.where(fixed.bool(), 1.0, d), 1e-13)


def _exact_batch(case, seed):
    systems, b, meshes, kappas = _batch(case["count"], case["side_min"], case["side_max"])
    rows, cols, vals, diag_fixed, group, n0 = [], [], [], [], [], 0
    for k, ((c, el), kap) in enumerate(zip(meshes, kappas)):
        X = torch.from_numpy(np.asarray(c)).to(DEV)
        e = torch.from_numpy(np.asarray(el)).to(DEV).long()
        G, w = _geometry("tri3", X[e])
        K = torch.einsum("eqad,eqbd,eq->eab", G, G, w) * torch.from_numpy(kap).to(DEV)[:, None, None]
        rows.append((e[:, :, None] + n0).expand(-1, 3, 3).reshape(-1))
        cols.append((e[:, None, :] + n0).expand(-1, 3, 3).reshape(-1))
        vals.append(K.reshape(-1))
        edge = ((X <= 1e-12) | (X >= 1 - 1e-12)).any(1)
        diag_fixed.append(edge)
        group.append(torch.full((X.shape[0],), k, device=DEV))
        n0 += X.shape[0]
    rows, cols, vals, edge, group = (torch.cat(t) for t in (rows, cols, vals, diag_fixed, group))
    vals = torch.where(edge[rows] | edge[cols], 0.0, vals)
    i = torch.arange(n0, device=DEV)
    M = torch.sparse_coo_tensor(torch.stack([torch.cat([rows, i]), torch.cat([cols, i])]),
                                torch.cat([vals, edge.double()]), (n0, n0)).coalesce()
    idx, val = M.indices(), M.values()
    d = torch.zeros(n0, dtype=torch.float64, device=DEV)
    on = idx[0] == idx[1]
    d[idx[0][on]] = val[on]
    M = M.to_sparse_csr()
    return _pcg(lambda x: M @ x, _batch_load(b, seed), 1.0 / d, 1e-13, group, len(meshes))


def exact(case, seed):
    fam = case["family"]
    if fam == "maps":
        return _exact_maps(case, seed)
    if fam == "energy":
        return _exact_state(case, seed, ("value", "residual"))
    if fam == "hvp":
        return _exact_state(case, seed, ("hvp",))
    if fam == "assemble":
        return _exact_state(case, seed, ("residual", "data"))
    mu, lam = LAWS["elastic"]
    if fam == "solve":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        c, _ = _mesh_arrays("hex8", nx, ny, nz, 0.0)
        fixed, load = _clamp(c, nx, ny, nz)
        return _exact_brick(nx, ny, nz, mu, lam, _solve_load(case, load, seed), fixed)
    if fam == "batch":
        return _exact_batch(case, seed)
    out = []
    for r in _requests(case, seed):
        if r.side > 32:  # minutes in plain torch, all together
            out.append(None)
            continue
        n = r.side
        c, _ = _mesh_arrays("hex8", n, n, n, 0.0)
        fixed, load = _clamp(c, n, n, n)
        mu_r = r.young / 2 / (1 + r.poisson)
        lam_r = r.young * r.poisson / (1 - 2 * r.poisson) / (1 + r.poisson)
        out.append(_exact_brick(n, n, n, mu_r, lam_r, load * r.traction, fixed))
    return out
