"""The calls a user of hyteg_b200 makes most, as cases that can be timed and compared.

A case names a path ("path"), a macro mesh ("mesh" with three counts "a", "b", "c" and a length "size"), a
refinement level and what else the path needs.  The macro meshes are boxes of a x b x c sub-cubes (six
tetrahedra each, `size` high) and spherical shells of the icosahedron (a: vertices per diamond edge, b:
radial layers of vertices, `size`: the inner radius).

prepare() builds what a program keeps over many calls: the storage, the operator (with stored element
matrices where the path uses them), the solver with its captured cycle, and the functions.  run() makes
one pass and returns the level vectors it wrote, as the library lays them out on the device.  exact()
computes the same in plain torch, in 64 bits, from the element integrals: micro-cells are visited one type
at a time, and nodes shared between macro-cells are found from their integer barycentric weights.
"""

import functools
import math

import numpy as np
import torch

import hyteg_b200 as H

RADIUS = {"p1": 2.2, "p2": 3.0}  # spectral radii given to the Chebyshev smoothers
RADIAL = (2.99, 1.0, 0.45)  # radial viscosity exp(a (r0 - |x|) / s)
PHASE = (0.125, 0.25, 0.0)
EXPSIN = 0.5
SHARE = {"float64": 8, "float32": 4, "float16": 2}
DTYPE = {"float64": torch.float64, "float32": torch.float32, "float16": torch.float16}


def listed():
    return [
        # the headline: one apply of the constant-stencil Laplacian on the unit cube, 17 M DoFs, vectors in HBM
        dict(name="p1 apply cube L8", path="p1_apply", mesh="box", a=1, b=1, c=1, size=1.0, level=8, dtype="float64"),
        # the same call on a small mesh, as the inner step of a Krylov method or a time step makes it: latency
        dict(name="p1 apply box L4 f32", path="p1_apply", mesh="box", a=3, b=2, c=1, size=1.0, level=4, dtype="float32"),
        # the small solve: ten V(2,2) weighted-Jacobi cycles on the level-5 cube with the residual of each cycle
        dict(name="p1 10 cycles cube L5", path="p1_solve", mesh="box", a=1, b=1, c=1, size=1.0, level=5, cycles=10, dtype="float64"),
        # one V(3,3) Chebyshev(3) cycle of the large cube, the step of a solve to a tight tolerance
        dict(name="p1 cycle cube L8", path="p1_cycle", mesh="box", a=1, b=1, c=1, size=1.0, level=8, dtype="float64"),
        # the single-precision smoother of a mixed-precision solve
        dict(name="p1 smooth box L7 f32", path="p1_smooth", mesh="box", a=2, b=1, c=1, size=1.0, level=7, steps=3, dtype="float32"),
        # variable coefficient on the blended shell with stored stencils: what a served solve runs per cycle
        dict(name="p1 div-k-grad cycle shell L5", path="p1k_cycle", mesh="shell", a=3, b=2, c=0, size=0.55, level=5, coeff="expsin", dtype="float64"),
        # linear transfers of one level pair, an odd box
        dict(name="p1 transfers box L7", path="p1_transfer", mesh="box", a=3, b=1, c=1, size=1.0, level=7, dtype="float64"),
        # quadratic elements with constant stencils
        dict(name="p2 apply cube L6", path="p2_apply", mesh="box", a=1, b=1, c=1, size=1.0, level=6, dtype="float64"),
        # the large matrix-free operator: quadratic elements, variable coefficient, blended shell
        dict(name="p2 div-k-grad shell L4", path="p2k_apply", mesh="shell", a=5, b=3, c=0, size=0.55, level=4, coeff="expsin", dtype="float64"),
        # Chebyshev smoothing of the same operator with stored element matrices, as its multigrid cycles run it
        dict(name="p2 smooth stored shell L4", path="p2k_smooth", mesh="shell", a=3, b=2, c=0, size=0.55, level=4, coeff="expsin", steps=1, dtype="float64"),
        # one Uzawa step of the Stokes multigrid, radial viscosity, stored velocity matrices
        dict(name="stokes uzawa shell L3", path="uzawa", mesh="shell", a=3, b=2, c=0, size=0.55, level=3, dtype="float64"),
        # the coupled full viscous block, matrix-free
        dict(name="full viscous shell L3", path="viscous", mesh="shell", a=3, b=3, c=0, size=0.55, level=3, coeff="radial", dtype="float64"),
    ]


def draw(rng):
    path = rng.choice(["p1_apply", "p1_apply", "p1_solve", "p1_cycle", "p1_smooth", "p1k_cycle", "p1_transfer", "p2_apply", "p2k_apply",
                       "p2k_smooth", "uzawa", "viscous"])
    box = path in ("p1_apply", "p1_solve", "p1_cycle", "p1_smooth", "p1_transfer", "p2_apply") or rng.random() < 0.25
    case = dict(path=path, mesh="box" if box else "shell", dtype="float64")
    if box:
        case.update(a=rng.randint(1, 4), b=rng.randint(1, 3), c=rng.randint(1, 3), size=round(rng.uniform(0.5, 2.0), 2))
        cells = 6 * case["a"] * case["b"] * case["c"]
    else:
        case.update(a=rng.choice([2, 3, 3, 5]), b=rng.randint(2, 3), c=0, size=round(rng.uniform(0.4, 0.7), 2))
        cells = 60 * (case["a"] - 1) ** 2 * (case["b"] - 1)
    lo, hi, most = {"p1_apply": (2, 8, 1.0e8), "p1_solve": (2, 6, 2.0e6), "p1_cycle": (3, 8, 1.0e8), "p1_smooth": (3, 8, 1.0e8),
                    "p1k_cycle": (2, 5, 8.0e6), "p1_transfer": (2, 8, 1.0e8), "p2_apply": (2, 7, 1.3e7), "p2k_apply": (1, 5, 8.0e6),
                    "p2k_smooth": (1, 5, 1.0e6), "uzawa": (1, 4, 1.3e5), "viscous": (1, 4, 5.0e5)}[path]
    fits = [l for l in range(lo, hi + 1) if cells * 8.0 ** l <= most] or [lo]
    case["level"] = rng.choice(fits[-5:])
    if path in ("p1_apply", "p1_smooth", "p1_transfer"):
        case["dtype"] = rng.choice(["float64", "float64", "float32", "float16"])
    elif path in ("p2k_apply", "p2_apply", "p2k_smooth"):
        case["dtype"] = rng.choice(["float64", "float64", "float32"])
    if path in ("p1_smooth", "p2k_smooth"):
        case["steps"] = rng.randint(1, 4)
    if path == "p1_solve":
        case["cycles"] = rng.randint(2, 10)
    if path in ("p1k_cycle", "p2k_apply", "p2k_smooth", "viscous"):
        case["coeff"] = rng.choice(["expsin", "expsin", "const"]) if box else rng.choice(["expsin", "radial", "const"])
    return case


# ------------------------------------------------------------------------------------------ macro meshes
def box_mesh(nx, ny, nz, height):
    """Sub-cubes (height `height`) split into the six tetrahedra around their main diagonal."""
    ids = np.arange((nx + 1) * (ny + 1) * (nz + 1)).reshape(nz + 1, ny + 1, nx + 1)
    coords = np.array([(x, y, z * height) for z in range(nz + 1) for y in range(ny + 1) for x in range(nx + 1)], dtype=float)
    cells = []
    for z in range(nz):
        for y in range(ny):
            for x in range(nx):
                for order in ((0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0)):
                    p, tet = [x, y, z], [ids[z, y, x]]
                    for d in order:
                        p[d] += 1
                        tet.append(ids[p[2], p[1], p[0]])
                    cells.append(tet)
    return coords, np.array(cells)


def shell_mesh(ntan, nrad, rmin):
    """The icosahedron's faces refined ntan - 1 times per edge, prisms between nrad radii, three tetrahedra
    per prism (split by the order of the vertex numbers, so that neighbours agree)."""
    g = (1 + math.sqrt(5)) / 2
    ico = np.array([(0, s, t * g) for s in (-1, 1) for t in (-1, 1)] + [(s, t * g, 0) for s in (-1, 1) for t in (-1, 1)] +
                   [(t * g, 0, s) for s in (-1, 1) for t in (-1, 1)])
    near = lambda i, j: abs(np.linalg.norm(ico[i] - ico[j]) - 2) < 1e-9  # noqa: E731
    faces = [(i, j, k) for i in range(12) for j in range(i) for k in range(j) if near(i, j) and near(j, k) and near(i, k)]
    m, ids, pts, tris = ntan - 1, {}, [], []

    def vid(p):
        p = p / np.linalg.norm(p)
        key = tuple(np.round(p, 9) + 0.0)
        if key not in ids:
            ids[key] = len(pts)
            pts.append(p)
        return ids[key]

    for f in faces:
        v = {(i, j): vid(ico[f[0]] * (m - i - j) + ico[f[1]] * i + ico[f[2]] * j) for i in range(m + 1) for j in range(m + 1 - i)}
        tris += [(v[i, j], v[i + 1, j], v[i, j + 1]) for i in range(m) for j in range(m - i)]
        tris += [(v[i + 1, j], v[i + 1, j + 1], v[i, j + 1]) for i in range(m) for j in range(m - i - 1)]
    n, radii = len(pts), np.linspace(rmin, 1.0, nrad)
    coords = np.concatenate([r * np.array(pts) for r in radii])
    cells = []
    for k in range(nrad - 1):
        for t in tris:
            a, b, c = sorted(t)
            a0, b0, c0, a1, b1, c1 = (x + n * (k + q) for q in (0, 1) for x in (a, b, c))
            cells += [(a0, b0, c0, c1), (a0, b0, b1, c1), (a0, a1, b1, c1)]
    return coords, np.array(cells)


@functools.lru_cache(maxsize=16)
def macro(mesh, a, b, c, size):
    coords, cells = box_mesh(a, b, c, size) if mesh == "box" else shell_mesh(a, b, size)
    return coords, np.array(sorted(map(tuple, cells)))


# ------------------------------------------------------------------------------------------ one level's layout
def up32(v):
    return (v + 31) // 32 * 32


def tet_points(n):
    """Points (x, y, z) of a macro-cell's array: x runs fastest, then y, then z."""
    z, y, x = torch.meshgrid(*(torch.arange(n + 1, device="cuda", dtype=torch.int32) for _ in range(3)), indexing="ij")
    keep = (x + y + z <= n).reshape(-1)
    return torch.stack([v.reshape(-1)[keep] for v in (x, y, z)], 1).long()


def cell_index(n, x, y, z):
    w, wz = n + 1, n + 1 - z
    return (w + 2) * (w + 1) * w // 6 - (wz + 2) * (wz + 1) * wz // 6 + y * (wz + 1) - y * (y + 1) // 2 + x


class Grid:
    """Node numbers of a level (shared nodes once) and their places in the library's vectors: every
    primitive's array in the order vertices, edges, faces, cells, on the device padded to 32 values."""

    def __init__(self, coords, cells, level):
        self.n = n = 1 << level
        self.coords, self.cells = torch.tensor(coords, device="cuda"), torch.tensor(cells, device="cuda")
        nv, nc = len(coords), len(cells)
        self.pts = tet_points(n)
        gen = np.random.RandomState(7)
        tag = torch.tensor(gen.randint(-2**62, 2**62, nv), device="cuda")
        w = torch.cat([n - self.pts.sum(1, keepdim=True), self.pts], 1)
        keys = torch.stack([sum(w[:, k] * tag[c[k]] for k in range(4)) for c in self.cells])
        uniq, gid = torch.unique(keys, return_inverse=True)
        self.gid, self.nodes = gid, uniq.numel()
        edges = np.unique(np.sort(np.concatenate([cells[:, [i, j]] for i in range(4) for j in range(i)]), axis=1), axis=0)
        tri = [np.sort(cells[:, f], axis=1) for f in ([1, 2, 3], [0, 2, 3], [0, 1, 3], [0, 1, 2])]  # opposite vertex 0..3
        faces, back, count = np.unique(np.concatenate(tri), axis=0, return_inverse=True, return_counts=True)
        back = back.reshape(4, nc)
        self.boundary = torch.zeros(self.nodes, dtype=torch.bool, device="cuda")
        for k in range(4):
            outer = torch.tensor(count[back[k]] == 1, device="cuda")
            self.boundary[gid[outer][:, w[:, k] == 0]] = True
        self.inner = ~self.boundary
        # array sizes per primitive: own points first, then layers of neighbours that only hold copies
        inc = lambda prim, what: np.array([sum(1 for q in what if set(p) <= set(q)) for p in prim.tolist()])  # noqa: E731
        ce, ct, cc = edges.tolist(), faces.tolist(), cells.tolist()
        tet, tr = (n + 3) * (n + 2) * (n + 1) // 6, (n + 2) * (n + 1) // 2
        low = (n + 2) * (n + 1) // 2 - (n + 1)
        fcells = count
        sizes = np.concatenate([1 + np.bincount(edges.reshape(-1), minlength=nv), (n + 1) + inc(edges, ct) * n + inc(edges, cc) * (n - 1),
                                tr + fcells * low, np.full(nc, tet)])
        del ce
        padded = up32(sizes)
        self.off = np.concatenate([[0], np.cumsum(padded)])
        self.poff = np.concatenate([[0], np.cumsum(sizes)])
        self.size, self.packed_size = int(self.off[-1]), int(self.poff[-1])
        # owners: (node, primitive, place in its array)
        node, prim, at = [], [], []

        def own(key, first, place):
            node.append(torch.searchsorted(uniq, key.reshape(-1)))
            prim.append((first + torch.arange(key.shape[0], device="cuda"))[:, None].expand(key.shape).reshape(-1))
            at.append(place[None, :].expand(key.shape).reshape(-1))

        own(n * tag[:, None], 0, torch.zeros(1, dtype=torch.long, device="cuda"))
        e, f = torch.tensor(edges, device="cuda"), torch.tensor(faces, device="cuda")
        i = torch.arange(1, n, device="cuda")
        if n > 1:
            own((n - i)[None] * tag[e[:, 0]][:, None] + i[None] * tag[e[:, 1]][:, None], nv, i)
        j, i = torch.meshgrid(torch.arange(1, n, device="cuda"), torch.arange(1, n, device="cuda"), indexing="ij")
        keep = i + j < n
        i, j = i[keep], j[keep]
        if i.numel():
            own((n - i - j)[None] * tag[f[:, 0]][:, None] + i[None] * tag[f[:, 1]][:, None] + j[None] * tag[f[:, 2]][:, None],
                nv + len(edges), j * (n + 2) - j * (j + 1) // 2 + i)
        self.own_node, self.own_prim, self.own_at = torch.cat(node), torch.cat(prim), torch.cat(at)
        self.first_cell, self.tet, self.nc = nv + len(edges) + len(faces), tet, nc

    def place(self, values, packed=False):
        """The level vector of node values (copies of neighbours in the lower primitives' arrays: zero)."""
        off = torch.tensor(self.poff if packed else self.off, device="cuda")
        out = torch.zeros(self.packed_size if packed else self.size, dtype=torch.float64, device="cuda")
        out[off[self.own_prim] + self.own_at] = values[self.own_node]
        start = off[self.first_cell:self.first_cell + self.nc]
        out[start[:, None] + torch.arange(self.tet, device="cuda")] = values[self.gid]
        return out

    def random(self, seed, k, dtype="float64", zero=None):
        """Uniform values in [-1, 1] per node as the storage type holds them; zero: nodes that are zero."""
        g = torch.Generator("cuda").manual_seed(seed * 64 + k)
        v = torch.rand(self.nodes, generator=g, device="cuda", dtype=torch.float64) * 2 - 1
        if zero is not None:
            v[zero] = 0
        return v.to(DTYPE[dtype]).double()


@functools.lru_cache(maxsize=12)
def grid_of(mesh, a, b, c, size, level):
    return Grid(*macro(mesh, a, b, c, size), level)


def mesh_of(case):
    return case["mesh"], case["a"], case["b"], case["c"], case["size"]


def grid(case, level):
    return grid_of(*mesh_of(case), level)


# ------------------------------------------------------------------------------------------ the library's side
def coefficient(case):
    kind = case.get("coeff", "const")
    return {"const": 1.5, "expsin": ("expsin", EXPSIN, PHASE), "radial": ("radial",) + RADIAL}[kind]


@functools.lru_cache(maxsize=1)
def context():
    """One context, and so one stream, for the program's life."""
    return H.Context(0)


class View:
    """A function's storage; the tensor made from it keeps the function alive."""

    def __init__(self, fn, ptr, n, code):
        self.fn = fn
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": (n,), "typestr": code, "version": 3}


def vector(state, fn, level):
    """The level's storage as a torch tensor, without a copy (views are kept by address and size)."""
    ptr, n = fn.device_ptr(level)
    key = (fn.name, ptr, n)
    if key not in state["views"]:
        state["views"][key] = torch.as_tensor(View(fn, ptr, n, {0: "<f8", 1: "<f4", 2: "<f2"}[fn.dtype]), device="cuda")
    return state["views"][key]


def prepare(case, seed):
    path, L, dt = case["path"], case["level"], case["dtype"]
    blend = "shell" if case["mesh"] == "shell" else None
    ctx = context()
    coords, cells = macro(*mesh_of(case))
    store = H.PrimitiveStorage.from_tets(coords, cells, ctx)
    s = dict(case=case, ctx=ctx, store=store, views={}, L=L)
    p2 = path in ("p2_apply", "p2k_apply", "p2k_smooth")
    kind = H.P2Function if p2 else H.P1Function
    g = grid(case, L + p2)
    cycle = path in ("p1_solve", "p1_cycle", "p1k_cycle")
    low = 0 if cycle else max(L - 1, 0)

    def fn(name, k=None, zero=None, lo=L, dtype=dt, kind=kind, gr=g):
        f = kind(name, store, lo, L, ctx, dtype)
        if k is not None:
            f.upload(L, gr.place(gr.random(seed, k, dtype, zero), packed=True).cpu().numpy())
        return f

    if path in ("p1_apply", "p2_apply", "p2k_apply"):
        s["op"] = {"p1_apply": lambda: H.P1ConstantLaplaceOperator(store, L, L, ctx), "p2_apply": lambda: H.P2ConstantLaplaceOperator(store, L, L, ctx),
                   "p2k_apply": lambda: H.P2ElementwiseBlendingDivKGradOperator(store, L, L, ctx, k=coefficient(case), blending=blend)}[path]()
        s["x"], s["y"] = fn("x", 1), fn("y")
        s["op"].apply(s["x"], s["y"], L, H.Inner)
    elif path == "viscous":
        g2 = grid(case, L + 1)
        s["op"] = H.P2ElementwiseBlendingFullViscousOperator(store, L, L, ctx, viscosity=coefficient(case), blending=blend)
        s["x"] = [fn("u%d" % k, 1 + k, kind=H.P2Function, gr=g2) for k in range(3)]
        s["y"] = [fn("v%d" % k, kind=H.P2Function) for k in range(3)]
        s["op"].apply(s["x"], s["y"], L, H.Inner)
    elif path == "p1_transfer":
        s["x"], s["r"], s["p"] = fn("x", 1, g.boundary, low), fn("r", None, None, low), fn("p", 2, g.boundary, low)
        s["R"], s["P"] = H.P1toP1LinearRestriction(), H.P1toP1LinearProlongation()
        s["p"].copyFrom(s["x"], L)
    elif cycle:
        if path == "p1k_cycle":
            s["op"] = H.P1ElementwiseBlendingDivKGradOperator(store, 0, L, ctx, k=coefficient(case), blending=blend)
            s["op"].computeAndStoreLocalElementMatrices()
        else:
            s["op"] = H.P1ConstantLaplaceOperator(store, 0, L, ctx)
        steps, smoother = (2, "jacobi") if path == "p1_solve" else (3, "chebyshev")
        s["mg"] = H.GeometricMultigridSolver(ctx, s["op"], 0, L, steps, steps, smoother=smoother)
        if smoother == "chebyshev":
            s["mg"].set_radii([RADIUS["p1"]] * (L + 1))
        s["x"], s["x0"], s["b"] = fn("x", None, None, 0), fn("x0", 1, g.boundary), fn("b", 2, g.boundary, 0)
        s["mg"].solve(s["op"], s["x"], s["b"], L)
    elif path in ("p1_smooth", "p2k_smooth"):
        if path == "p1_smooth":
            s["op"] = H.P1ConstantLaplaceOperator(store, low, L, ctx)
        else:
            s["op"] = H.P2ElementwiseBlendingDivKGradOperator(store, low, L, ctx, k=coefficient(case), blending=blend)
            s["op"].computeAndStoreLocalElementMatrices()
        s["mg"] = H.GeometricMultigridSolver(ctx, s["op"], low, L, smoother="chebyshev")
        s["mg"].set_radii([RADIUS["p1" if path == "p1_smooth" else "p2"]] * (L - low + 1))
        s["x"], s["x0"], s["b"] = fn("x", None, None, low), fn("x0", 1, g.boundary), fn("b", 2, g.boundary, low)
        s["mg"].smooth(s["x"], s["b"], L, 1)
    elif path == "uzawa":
        g2 = grid(case, L + 1)
        s["st"] = H.StokesUzawaMultigrid(ctx, store, low, L, viscosity=("radial",) + RADIAL, blending=blend, omega=0.7,
                                         pressure_scaling="lumped_mass")
        s["st"].set_velocity_radii([RADIUS["p2"]] * (L - low + 1))
        for k in range(3):
            s["u%d" % k] = fn("u%d" % k, None, None, low, kind=H.P2Function)
            s["w%d" % k] = fn("w%d" % k, 1 + k, g2.boundary, kind=H.P2Function, gr=g2)
            s["b%d" % k] = fn("b%d" % k, 4 + k, g2.boundary, low, kind=H.P2Function, gr=g2)
        s["p"], s["p0"], s["bp"] = fn("p", None, None, low), fn("p0", 7), fn("bp", 8, None, low)
        s["u"], s["bu"] = [s["u%d" % k] for k in range(3)], [s["b%d" % k] for k in range(3)]
        s["st"].uzawa_smooth(s["u"], s["p"], s["bu"], s["bp"], L)
    ctx.synchronize()
    return s


def run(s):
    case, L = s["case"], s["L"]
    path = case["path"]
    if path in ("p1_apply", "p2_apply", "p2k_apply"):
        s["op"].apply(s["x"], s["y"], L, H.Inner)
        return vector(s, s["y"], L)
    if path == "viscous":
        s["op"].apply(s["x"], s["y"], L, H.Inner)
        return [vector(s, v, L) for v in s["y"]]
    if path == "p1_transfer":
        # residual down, correction of the coarser level up
        s["R"].restrict(s["x"], L, H.Inner)
        s["p"].copyFrom(s["x"], L)
        s["p"].copyFrom(s["x"], L - 1)
        s["P"].prolongateAndAdd(s["p"], L - 1, H.Inner)
        return [vector(s, s["x"], L - 1), vector(s, s["p"], L)]
    if path == "uzawa":
        for k in range(3):
            s["u"][k].copyFrom(s["w%d" % k], L)
        s["p"].copyFrom(s["p0"], L)
        s["st"].uzawa_smooth(s["u"], s["p"], s["bu"], s["bp"], L)
        return [vector(s, v, L) for v in s["u"] + [s["p"]]]
    # a solve from the caller's guess
    s["x"].copyFrom(s["x0"], L)
    if path == "p1_solve":
        history = s["mg"].solve_cycles(s["x"], s["b"], L, case["cycles"])
        return [vector(s, s["x"], L), history]
    if path in ("p1_smooth", "p2k_smooth"):
        s["mg"].smooth(s["x"], s["b"], L, case["steps"])
    else:
        s["mg"].solve(s["op"], s["x"], s["b"], L)
    return vector(s, s["x"], L)


def work(case):
    """Vectors once in and once out, and per stored matrix its distinct entries once."""
    path, L = case["path"], case["level"]
    cells = len(macro(*mesh_of(case))[1])
    micro = cells * 8.0 ** L
    dof, b = micro / 6, SHARE[case["dtype"]]  # P1 nodes; P2 nodes of the level: eight times as many
    if path == "p1_apply":
        return {"bytes": 2 * b * dof, "flops": 29 * dof}
    if path == "p2_apply":
        return {"bytes": 16 * b * dof, "flops": 8 * 56.5 * dof}
    if path == "p2k_apply":
        # per point of the eleven: the mapped gradient both ways and the coefficient, about 200 operations
        return {"bytes": 16 * b * dof, "flops": 2200.0 * micro}
    if path == "viscous":
        return {"bytes": 48 * b * dof, "flops": 1500.0 * micro}
    if path == "p1_transfer":
        return {"bytes": (2 + 1.0 / 8) * b * dof, "flops": 12 * dof}
    sweeps = {"p1_solve": 5 * case.get("cycles", 1), "p1_cycle": 19, "p1k_cycle": 19, "p1_smooth": 3 * case.get("steps", 1)}
    if path in sweeps:
        k = sweeps[path] * (1 if path == "p1_smooth" else 8.0 / 7)
        matrix = 8.0 * b * dof if path == "p1k_cycle" else 0  # 15 weights, symmetric
        return {"bytes": k * (3 * b * dof + matrix), "flops": k * 32 * dof}
    matrix = 8 * 15.0 * b * dof  # 28.75 entries per P2 node on average, symmetric
    if path == "p2k_smooth":
        return {"bytes": 3 * case["steps"] * (24 * b * dof + matrix), "flops": 3 * case["steps"] * 8 * 60 * dof}
    return {"bytes": 9 * (72 * b * dof + matrix), "flops": 27 * 8 * 60 * dof + 800.0 * micro}


def tolerance(case):
    """About four times and more what the paths differ by from exact(): 2e-14, 1.3e-7 and 3e-4 of the 2-norm."""
    return {"float64": {"rel": 2e-13}, "float32": {"rel": 1e-6}, "float16": {"rel": 2e-3}}[case["dtype"]]


# ------------------------------------------------------------------------------------------ in plain torch
TYPES = (((0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1)), ((1, 0, 0), (1, 1, 0), (0, 1, 0), (1, 0, 1)), ((1, 0, 0), (0, 1, 0), (1, 0, 1), (0, 0, 1)),
         ((1, 1, 0), (1, 1, 1), (0, 1, 1), (1, 0, 1)), ((1, 0, 1), (0, 1, 1), (0, 0, 1), (0, 1, 0)), ((0, 1, 0), (1, 1, 0), (1, 0, 1), (0, 1, 1)))
EDGES = ((2, 3), (1, 3), (1, 2), (0, 3), (0, 2), (0, 1))
LAMBDA = np.array([[-1.0, -1.0, -1.0], [1.0, 0.0, 0.0], [0.0, 1.0, 0.0], [0.0, 0.0, 1.0]])
# the 11 points of a rule of degree four (Xiao and Gimbutas), barycentric; its weights follow from its degree
POINTS11 = np.array([[0.17469405869723054, 0.04049050672759043, 0.01356070187980288, 0.7712547326953761],
                     [0.08140491840285922, 0.752508507009655, 0.06809937093820666, 0.09798720364927911],
                     [0.3044484024344971, 0.2402766649280726, 0.126801725915392, 0.3284732067220384],
                     [0.7412288820936226, 0.0672232948933834, 0.03518392977359872, 0.1563638932393953],
                     [0.053341239535745266, 0.419266313879513, 0.04778143555908666, 0.4796110110256551],
                     [0.4329534904813558, 0.4507658760912768, 0.05945661629943383, 0.05682401712793367],
                     [0.5380072039161857, 0.1294113737889104, 0.3301904148374645, 0.002391007457439365],
                     [0.008991260093335729, 0.1215419913339278, 0.3064939884296903, 0.5629727601430461],
                     [0.10660417256199362, 0.09720464458758327, 0.68439041545304, 0.1118007673973831],
                     [0.3292329597426468, 0.02956949520647961, 0.3179035602133946, 0.323293984837479],
                     [0.10384411641099309, 0.4327102390477686, 0.3538232392092971, 0.1096224053319412]])[:, 1:]


def rule(name):
    if name == "one":
        return np.full((1, 3), 0.25), np.array([1 / 6])
    if name == "four":
        a, b = (5 - math.sqrt(5)) / 20, (5 + 3 * math.sqrt(5)) / 20
        return np.array([[a, a, a], [b, a, a], [a, b, a], [a, a, b]]), np.full(4, 1 / 24)
    if name == "five":
        c = 1 / 6
        return np.array([[0.25, 0.25, 0.25], [c, c, c], [0.5, c, c], [c, 0.5, c], [c, c, 0.5]]), np.array([-2 / 15] + [3 / 40] * 4)
    f, rows, rhs = math.factorial, [], []
    for i in range(5):
        for j in range(5 - i):
            for k in range(5 - i - j):
                rows.append(POINTS11[:, 0] ** i * POINTS11[:, 1] ** j * POINTS11[:, 2] ** k)
                rhs.append(f(i) * f(j) * f(k) / f(i + j + k + 3))
    return POINTS11, np.linalg.lstsq(np.array(rows), np.array(rhs), rcond=None)[0]


def gradients(order, xi):
    lam = np.array([1 - xi.sum(), *xi])
    if order == 1:
        return LAMBDA
    return np.concatenate([(4 * lam - 1)[:, None] * LAMBDA, [4 * (lam[i] * LAMBDA[j] + lam[j] * LAMBDA[i]) for i, j in EDGES]])


def micro_cells(case, level, order, most=400_000):
    """(macro-cells, node numbers [C, M, 4 or 10], vertices [C, M, 4, 3]) in pieces."""
    gr = grid(case, level + (order == 2))
    n, step = 1 << level, order
    base = tet_points(n)
    for off in TYPES:
        shift = max(sum(o) for o in off) - 1
        a = base[base.sum(1) <= n - 1 - shift]
        if not a.numel():
            continue
        V = [a + torch.tensor(o, device="cuda") for o in off]
        nodes = [step * v for v in V] + ([V[i] + V[j] for i, j in EDGES] if order == 2 else [])
        idx = torch.stack([cell_index(gr.n, v[:, 0], v[:, 1], v[:, 2]) for v in nodes], 1)
        per = max(1, most // len(a))
        for c0 in range(0, gr.nc, per):
            cs = slice(c0, min(gr.nc, c0 + per))
            P = gr.coords[gr.cells[cs]]
            ax = (P[:, 1:] - P[:, :1]) / n
            X = torch.stack([P[:, None, 0] + torch.einsum("mk,ckd->cmd", v.double(), ax) for v in V], 2)
            yield cs, gr.gid[cs][:, idx], X


def vertices1(case, level):
    """Node numbers of the micro-cells' vertices on the level itself, in the order of micro_cells()."""
    for cs, ids, _ in micro_cells(case, level, 1):
        yield ids


def mapped(case, cs, X, xi, coeff):
    """At one point of every micro-cell: inverse Jacobian of the blended map, |det|, coefficient."""
    J = (X[:, :, 1:] - X[:, :, :1]).transpose(2, 3)
    P = X[:, :, 0] + J @ torch.tensor(xi, device="cuda")
    M, F = J, P
    if case["mesh"] == "shell":
        # the blended point keeps its direction and takes the radius of its layer: an affine function of the
        # point that is |v| at the vertices of the cell's layer triangles
        n = layer_normal(case)[cs]
        r, R = P.norm(dim=-1), torch.einsum("cmd,cd->cm", P, n)
        F = P * (R / r)[..., None]
        grad = n[:, None] / r[..., None] - P * (R / r**3)[..., None]
        M = ((R / r)[..., None, None] * torch.eye(3, device="cuda", dtype=torch.float64) + P[..., :, None] * grad[..., None, :]) @ J
    k = 1.0
    if coeff == "const":
        k = 1.5
    elif coeff == "expsin":
        t = 2 * math.pi * (F + torch.tensor(PHASE, device="cuda", dtype=torch.float64))
        k = torch.exp(EXPSIN * torch.sin(t[..., 0]) * torch.cos(t[..., 1]) * torch.sin(t[..., 2]))
    elif coeff == "radial":
        k = torch.exp(RADIAL[0] * (RADIAL[1] - F.norm(dim=-1)) / RADIAL[2])
    c = torch.linalg.cross
    m0, m1, m2 = M[..., 0], M[..., 1], M[..., 2]
    c0, c1, c2 = c(m1, m2), c(m2, m0), c(m0, m1)
    det = (m0 * c0).sum(-1)
    return torch.stack([c0, c1, c2], -2) / det[..., None, None], det.abs(), k


def layer_normal(case):
    """Per macro-cell of a shell the n with n . v = |v| at its vertices (two parallel triangles)."""
    coords, cells = macro(*mesh_of(case))
    V = coords[cells]
    return torch.tensor(np.stack([np.linalg.lstsq(v, np.linalg.norm(v, axis=1), rcond=None)[0] for v in V]), device="cuda")


class Matrix:
    """The operator of a level as its micro-cells' matrices, summed over shared nodes; rows that are not
    flagged are zero."""

    def __init__(self, case, level, order, coeff, points):
        self.gr = grid(case, level + (order == 2))
        self.parts = []
        plain = coeff is None and case["mesh"] == "box"
        for cs, ids, X in micro_cells(case, level, order):
            Y = X[:, :1] if plain else X  # affine and constant: one matrix per macro-cell and type
            K = 0
            for xi, w in zip(*rule(points)):
                Mi, det, k = mapped(case, cs, Y, xi, coeff)
                G = torch.tensor(gradients(order, xi), device="cuda") @ Mi
                K = K + (w * det * k)[..., None, None] * (G @ G.transpose(-1, -2))
            self.parts.append((ids, K))
        self.diag = torch.zeros(self.gr.nodes, dtype=torch.float64, device="cuda")
        for ids, K in self.parts:
            d = K.diagonal(dim1=-2, dim2=-1).expand(ids.shape)
            self.diag.index_add_(0, ids.reshape(-1), d.reshape(-1))

    def __call__(self, x, rows):
        y = torch.zeros_like(x)
        for ids, K in self.parts:
            xl = x[ids]
            yl = xl @ K.transpose(-1, -2)[:, 0] if K.shape[1] == 1 else (K @ xl[..., None])[..., 0]
            y.index_add_(0, ids.reshape(-1), yl.reshape(-1))
        return y * rows

    def dense(self):
        D = torch.zeros(self.gr.nodes**2, dtype=torch.float64, device="cuda")
        for ids, K in self.parts:
            at = ids[..., :, None] * self.gr.nodes + ids[..., None, :]
            D.index_add_(0, at.reshape(-1), K.expand(at.shape).reshape(-1))
        return D.reshape(self.gr.nodes, -1)


def chebyshev(A, x, b, radius, rows):
    """x + p(D^-1 A) D^-1 (b - A x) with 1 - t p(t) the scaled Chebyshev polynomial of degree three on
    [0.3, 1.2] times the radius."""
    lo, hi = 0.3 * radius, 1.2 * radius
    T = np.polynomial.chebyshev.Chebyshev([0, 0, 0, 1], domain=[lo, hi]).convert(kind=np.polynomial.Polynomial).coef
    c = -T[1:] / np.polynomial.polynomial.polyval(0.0, T)
    z = (b - A(x, rows)) / A.diag * rows
    x = x + c[0] * z
    for k in (1, 2):
        z = A(z, rows) / A.diag * rows
        x = x + c[k] * z
    return x


def prolongation(case, level):
    """Per node of `level` its two nodes of level - 1 (the same node twice where it is one of them)."""
    f, c = grid(case, level), grid(case, level - 1)
    p, odd = f.pts, f.pts % 2
    first = {(1, 0, 0): (1, 0, 0), (0, 1, 0): (0, 1, 0), (0, 0, 1): (0, 0, 1), (1, 1, 0): (1, -1, 0), (1, 0, 1): (1, 0, -1), (0, 1, 1): (0, 1, -1),
             (1, 1, 1): (1, -1, 1)}
    d = torch.zeros_like(p)
    for k, v in first.items():
        d[(odd == torch.tensor(k, device="cuda")).all(1)] = torch.tensor(v, device="cuda")
    # both ends as one macro-cell sees them (cells may see an edge from either side)
    one = torch.empty(f.nodes, dtype=torch.long, device="cuda")
    one[f.gid.reshape(-1)] = torch.arange(f.gid.numel(), device="cuda")
    cell, at = one // len(p), one % len(p)
    ends = []
    for q in ((p + d) // 2, (p - d) // 2):
        ends.append(c.gid[cell, cell_index(c.n, q[:, 0], q[:, 1], q[:, 2])[at]])
    return ends


def restrict(case, level, x):
    a, b = prolongation(case, level)
    y = torch.zeros(grid(case, level - 1).nodes, dtype=torch.float64, device="cuda")
    same = a == b
    y.index_add_(0, a, torch.where(same, x, 0.5 * x))
    y.index_add_(0, b, torch.where(same, 0 * x, 0.5 * x))
    return y


def prolong(case, level, x):
    a, b = prolongation(case, level)
    return torch.where(a == b, x[a], 0.5 * (x[a] + x[b]))


def v_cycle(case, ops, smooth, steps, x, b, level):
    A, gr = ops[level], grid(case, level)
    rows = gr.inner.double()
    if level == 0:
        i = torch.nonzero(gr.inner)[:, 0]
        if i.numel():
            x = x.clone()
            x[i] = torch.linalg.solve(A.dense()[i][:, i], b[i])
        return x
    for _ in range(steps):
        x = smooth(A, x, b, rows)
    coarse = grid(case, level - 1)
    r = restrict(case, level, (b - A(x, rows)) * rows) * coarse.inner
    e = v_cycle(case, ops, smooth, steps, torch.zeros_like(r), r, level - 1)
    x = x + prolong(case, level, e) * rows
    for _ in range(steps):
        x = smooth(A, x, b, rows)
    return x


def exact(case, seed):
    path, L, dt = case["path"], case["level"], case["dtype"]
    coeff = case.get("coeff")
    if path == "p1_transfer":
        f, c = grid(case, L), grid(case, L - 1)
        x = f.random(seed, 1, dt, f.boundary)
        r = restrict(case, L, x) * c.inner
        return [c.place(r), f.place(x + prolong(case, L, r.to(DTYPE[dt]).double()) * f.inner)]
    order = 2 if path in ("p2_apply", "p2k_apply", "p2k_smooth", "viscous", "uzawa") else 1
    gr = grid(case, L + (order == 2))
    rows = gr.inner.double()
    if path in ("p1_apply", "p2_apply", "p2k_apply"):
        A = Matrix(case, L, order, coeff, {"p1_apply": "one", "p2_apply": "four", "p2k_apply": "eleven"}[path])
        return gr.place(A(gr.random(seed, 1, dt), rows))
    if path in ("p1_smooth", "p2k_smooth"):
        A = Matrix(case, L, order, coeff, "one" if path == "p1_smooth" else "eleven")
        x, b = gr.random(seed, 1, dt, gr.boundary), gr.random(seed, 2, dt, gr.boundary)
        for _ in range(case["steps"]):
            x = chebyshev(A, x, b, RADIUS["p1" if path == "p1_smooth" else "p2"], rows)
        return gr.place(x)
    if path in ("p1_solve", "p1_cycle", "p1k_cycle"):
        ops = [Matrix(case, l, 1, coeff, "five" if path == "p1k_cycle" else "one") for l in range(L + 1)]
        x, b = gr.random(seed, 1, dt, gr.boundary), gr.random(seed, 2, dt, gr.boundary)
        if path != "p1_solve":
            return gr.place(v_cycle(case, ops, lambda A, x, b, m: chebyshev(A, x, b, RADIUS["p1"], m), 3, x, b, L))
        jacobi = lambda A, x, b, m: x + (2 / 3) * (b - A(x, m)) / A.diag * m  # noqa: E731
        norm = lambda x: ((b - ops[L](x, rows)) * rows).norm().item()  # noqa: E731
        history = [norm(x)]
        for _ in range(case["cycles"]):
            x = v_cycle(case, ops, jacobi, 2, x, b, L)
            history.append(norm(x))
        return [gr.place(x), np.array(history)]
    if path == "viscous":
        u = [gr.random(seed, 1 + k, dt) for k in range(3)]
        out = [torch.zeros_like(v) for v in u]
        for cs, ids, X in micro_cells(case, L, 2):
            ul = torch.stack([v[ids] for v in u], -1)
            y = torch.zeros_like(ul)
            for xi, w in zip(*rule("five")):
                Mi, det, mu = mapped(case, cs, X, xi, coeff)
                G = torch.tensor(gradients(2, xi), device="cuda") @ Mi
                D = ul.transpose(-1, -2) @ G
                S = D + D.transpose(-1, -2) - (2 / 3) * D.diagonal(dim1=-2, dim2=-1).sum(-1)[..., None, None] * torch.eye(3, device="cuda")
                y += (w * mu * det)[..., None, None] * (G @ S.transpose(-1, -2))
            for k in range(3):
                out[k].index_add_(0, ids.reshape(-1), y[..., k].reshape(-1))
        return [gr.place(v * rows) for v in out]
    # the Uzawa step: velocity smoothing with b - B^T p, then the pressure update
    pg = grid(case, L)
    A = Matrix(case, L, 2, "radial", "eleven")
    u = [gr.random(seed, 1 + k, dt, gr.boundary) for k in range(3)]
    b = [gr.random(seed, 4 + k, dt, gr.boundary) for k in range(3)]
    p, bp = pg.random(seed, 7, dt), pg.random(seed, 8, dt)
    blocks, scale = [], torch.zeros(pg.nodes, dtype=torch.float64, device="cuda")
    pieces = list(zip(micro_cells(case, L, 2), vertices1(case, L)))
    for (cs, ids, X), ip in pieces:
        B = 0
        for xi, w in zip(*rule("four")):
            Mi, det, _ = mapped(case, cs, X, xi, None)
            lam = torch.tensor([1 - xi.sum(), *xi], device="cuda")
            G = torch.tensor(gradients(2, xi), device="cuda") @ Mi
            B = B - (w * det)[..., None, None, None] * lam[:, None, None] * G[..., None, :, :]  # [C, M, 4, 10, 3]
        blocks.append((ids, ip, B))
        for xi, w in zip(*rule("five")):
            _, det, eta = mapped(case, cs, X, xi, "radial")
            lam = torch.tensor([1 - xi.sum(), *xi], device="cuda")
            scale.index_add_(0, ip.reshape(-1), (-(w * det / eta)[..., None] * lam).reshape(-1))
    r = [v.clone() for v in b]
    for ids, ip, B in blocks:
        t = torch.einsum("cmijd,cmi->cmjd", B, p[ip])
        for k in range(3):
            r[k].index_add_(0, ids.reshape(-1), -t[..., k].reshape(-1))
    for k in range(3):
        for _ in range(3):
            u[k] = chebyshev(A, u[k], r[k] * rows, RADIUS["p2"], rows)
    rp = bp.clone()
    for ids, ip, B in blocks:
        t = torch.einsum("cmijd,cmjd->cmi", B, torch.stack([v[ids] for v in u], -1))
        rp.index_add_(0, ip.reshape(-1), -t.reshape(-1))
    return [gr.place(v) for v in u] + [pg.place(p + 0.7 * rp / scale)]
