"""P1 constant-stencil operations at the levels around the change from the one-launch kernel (up to 64 points
per macro-edge) to the tiled sweeps, and on meshes with edges and vertices of many cells: apply, add, Jacobi
step and Chebyshev step, with Neumann faces (one cell), against the oracle's assembled operator in FP64 (1e-12
of the largest value as in the other P1 tests); what every operation does to unflagged owners."""

import ctypes

import numpy as np
import pytest

import hyteg_b200 as H
from oracle import hyteg_oracle as O
from tests import meshes as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh", ["unit_tet", "pyramid_4", "octahedron_8", "cube_2x1x1"])
@pytest.mark.parametrize("L", [0, 1, 2, 4])
@pytest.mark.parametrize("neumann", [False, True])
def test_p1_operations(ctx, mesh, L, neumann):
    coords, tets = M.ALL[mesh]()
    om = O.MacroMesh(coords, tets, bc_types={0: O.INNER, 1: O.NEUMANN} if neumann else None)
    op = O.P1ConstantLaplace(om, L, L)
    lev = op.levels[L]
    pm = H.PrimitiveStorage.from_tets(coords, tets, ctx)
    if neumann:
        pm.set_bc_type(1, H.NeumannBoundary)
    A = H.P1ConstantLaplaceOperator(pm, L, L, ctx)
    flag = H.Inner | H.NeumannBoundary
    rng = np.random.default_rng(L)
    vec = {}
    for n in ("x", "b", "y"):
        v = np.zeros(lev.size)
        v[lev.owned] = rng.uniform(-1, 1, lev.owned.size)
        vec[n] = lev.sync(v)
    f = {n: H.P1Function(n, pm, L, L, ctx) for n in vec}
    for n in vec:
        f[n].upload(L, vec[n])
    own = lev.owned_mask(O.ALL)

    def check(got, ref):
        assert np.abs(got[own] - ref[own]).max() <= 1e-12 * max(np.abs(ref[own]).max(), 1e-300)
        d, s = lev.copy_map()
        np.testing.assert_array_equal(got[d], got[s])

    A.apply(f["x"], f["y"], L, flag)
    ref = op.apply(vec["x"], vec["y"].copy(), L, flag)
    check(f["y"].download(L), ref)
    A.apply(f["x"], f["y"], L, flag, H.Add)
    check(f["y"].download(L), op.apply(vec["x"], lev.sync(ref.copy()), L, flag, add=True))
    A.smooth_jac(f["y"], f["b"], f["x"], 0.6, L, flag)
    jac = op.smooth_jac(lev.sync(op.apply(vec["x"], lev.sync(ref.copy()), L, flag, add=True)), vec["b"], vec["x"], 0.6, L, flag)
    check(f["y"].download(L), jac)


def _shell(ntan, nrad):
    return lambda: O.mesh_spherical_shell(ntan, nrad, 0.55, 1.0)


# both sides of the changes between one thread per point and the tiles, by points per edge (64 and 128) and at 32
# and 64 by the level's points: 60, 120 and 240 cells of 64 points have 2.4, 4.8 and 9.5 million, 960 of 32 have 4.3
SIZES = {"cube 5": (M.cube_6, 5), "cube 6": (M.cube_6, 6), "cube 7": (M.cube_6, 7), "60 cells 6": (_shell(2, 2), 6),
         "120 cells 6": (_shell(2, 3), 6), "240 cells 6": (_shell(3, 2), 6), "960 cells 5": (_shell(5, 2), 5)}


@pytest.mark.parametrize("size", sorted(SIZES))
@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_p1_apply_across_kernels(ctx, size, dtype):
    """The constant stencils against the elementwise operator with k = 1 in FP64 (the same matrix; 1e-12 of the
    largest value, FP32 15 products per cell and up to 30 cells: 64 eps)."""
    make, L = SIZES[size]
    coords, tets = make()
    pm = H.PrimitiveStorage.from_tets(coords, tets, ctx)
    C = H.P1ConstantLaplaceOperator(pm, L, L, ctx)
    E = H.P1ElementwiseBlendingDivKGradOperator(pm, L, L, ctx, k=1.0)
    x, y = (H.P1Function(n, pm, L, L, ctx, dtype) for n in "xy")
    u, z = (H.P1Function(n, pm, L, L, ctx) for n in "uz")
    x.fill_random(L, 7)
    u.upload(L, x.download(L).astype(np.float64))
    for update in (H.Replace, H.Add):
        C.apply(x, y, L, H.Inner, update)
        E.apply(u, z, L, H.Inner, update)
        a, b = y.download(L), z.download(L)
        assert np.abs(a - b).max() <= (1e-12 if dtype == "float64" else 8e-6) * np.abs(b).max()


@pytest.mark.parametrize("size", sorted(SIZES))
@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_p1_chebyshev_across_kernels(ctx, size, dtype):
    """One Chebyshev(3) step equals its definition from the operator's own apply (FP64 1e-12; FP32: three
    applies of 15 products each, values up to 10: 200 eps)."""
    make, L = SIZES[size]
    coords, tets = make()
    pm = H.PrimitiveStorage.from_tets(coords, tets, ctx)
    A = H.P1ConstantLaplaceOperator(pm, L - 1, L, ctx)
    g = H.GeometricMultigridSolver(ctx, A, L - 1, L, smoother="chebyshev")
    g.set_radii([2.0, 2.0])
    c = H.chebyshev_coefficients(3, 0.3 * 2.0, 1.2 * 2.0)
    f = {n: H.P1Function(n, pm, L - 1, L, ctx, dtype) for n in ("x", "b", "r", "z", "t", "d", "ref")}
    for n in ("x", "b"):
        f[n].fill_random(L, 5 if n == "x" else 6)
        f[n].interpolate(0.0, L, H.DirichletBoundary)
    A.getInverseDiagonalValues(f["d"], L, H.Inner)
    f["ref"].copyFrom(f["x"], L)
    A.apply(f["x"], f["t"], L, H.Inner)
    f["r"].assign([1.0, -1.0], [f["b"], f["t"]], L, H.Inner)
    f["z"].multElementwise([f["d"], f["r"]], L, H.Inner)
    f["ref"].add([c[0]], [f["z"]], L, H.Inner)
    for k in (1, 2):
        A.apply(f["z"], f["t"], L, H.Inner)
        f["z"].multElementwise([f["d"], f["t"]], L, H.Inner)
        f["ref"].add([c[k]], [f["z"]], L, H.Inner)
    g.smooth(f["x"], f["b"], L, 1)
    x, ref = f["x"].download(L), f["ref"].download(L)
    assert np.abs(x - ref).max() <= (1e-12 if dtype == "float64" else 2.4e-5) * np.abs(ref).max()


@pytest.mark.parametrize("L", [1, 4, 7])
@pytest.mark.parametrize("p2", [False, True])
def test_unflagged_owners_are_carried_or_left(ctx, L, p2):
    """Dirichlet owners and their copies under flag Inner, all with nonzero values: Jacobi and the first Chebyshev
    step carry src over, the middle step the iterate; every other operation leaves its target as it was, whether
    or not the caller asks for a copy."""
    coords, tets = M.octahedron_8() if L < 7 else M.cube_6()
    pm = H.PrimitiveStorage.from_tets(coords, tets, ctx)
    L -= 1 if p2 else 0  # the same points per macro-edge
    A = (H.P2ConstantLaplaceOperator if p2 else H.P1ConstantLaplaceOperator)(pm, L, L, ctx)
    kind = H.P2Function if p2 else H.P1Function
    f = {n: kind(n, pm, L, L, ctx) for n in ("src", "v1", "v2", "dst", "mask")}
    f["mask"].interpolate(0.0, L, H.All)
    f["mask"].interpolate(1.0, L, H.DirichletBoundary)
    dirichlet = f["mask"].download(L) == 1.0
    assert dirichlet.any()
    raw = H.lib().hyb_internal_op_stencil
    raw.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_uint32, ctypes.c_int] + [ctypes.c_void_p] * 4 + [ctypes.c_double] * 2
    carried = {3: "src", 4: "src", 5: "v2"}  # Jacobi, first and middle Chebyshev step
    for code in range(8):
        for copy in (0, 1):
            before = {}
            for i, n in enumerate(("src", "v1", "v2", "dst")):
                f[n].fill_random(L, 10 * code + i)
                f[n].add([1.0 if n != "dst" else 3.0], [f["mask"]], L, H.DirichletBoundary)
                before[n] = f[n].download(L)
            assert raw(A.h, L, code, H.Inner, copy, *(f[n].h for n in ("src", "v1", "v2", "dst")), 0.5, 0.25) == 0
            want = before[carried[code]] if copy and code in carried else before["dst"]
            np.testing.assert_array_equal(f["dst"].download(L)[dirichlet], want[dirichlet], err_msg=f"dst of operation {code}, copy {copy}")
            np.testing.assert_array_equal(f["v2"].download(L)[dirichlet], before["v2"][dirichlet], err_msg=f"v2 of operation {code}, copy {copy}")


@pytest.mark.parametrize("L", [3, 6, 7])
@pytest.mark.parametrize("smoother", ["jacobi", "chebyshev"])
def test_smoothers_keep_boundary_values(ctx, L, smoother):
    """A smoothing step returns nonzero Dirichlet values unchanged at owners and copies."""
    coords, tets = M.cube_6()
    pm = H.PrimitiveStorage.from_tets(coords, tets, ctx)
    A = H.P1ConstantLaplaceOperator(pm, L - 1, L, ctx)
    g = H.GeometricMultigridSolver(ctx, A, L - 1, L, smoother=smoother)
    if smoother == "chebyshev":
        g.set_radii([2.0, 2.0])
    x, b, mask = (H.P1Function(n, pm, L - 1, L, ctx) for n in ("x", "b", "mask"))
    x.fill_random(L, 1)
    b.fill_random(L, 2)
    mask.interpolate(0.0, L, H.All)
    mask.interpolate(1.0, L, H.DirichletBoundary)
    x.add([2.0], [mask], L, H.DirichletBoundary)
    dirichlet, before = mask.download(L) == 1.0, x.download(L)
    for _ in range(2):
        g.smooth(x, b, L, 1)
    after = x.download(L)
    np.testing.assert_array_equal(after[dirichlet], before[dirichlet])
    assert (after != before).any()
