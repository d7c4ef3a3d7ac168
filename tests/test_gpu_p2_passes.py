"""Matrix-free P2 passes at the sizes where their blocks and node windows end: levels 0 and 1 (one anchor
per parity class, windows cut by the slanted face), level 4 of one tetrahedron (more anchors per class than
a block holds), every coefficient kind, with and without the shell map, against the oracle's element
matrices.  FP64 within 1e-12 of the largest value, the tolerance of the other P2 tests; FP32 sums about
300 rounded terms per node, so 300 eps = 4e-5 bounds it."""

import numpy as np
import pytest

import hyteg_b200 as H
from oracle import hyteg_oracle as O
from tests import meshes as M
from tests.test_gpu_p2 import _rand, _relerr

pytestmark = pytest.mark.gpu

SPECS = {"const": (1.75, lambda P: np.full(np.asarray(P).shape[:-1], 1.75)),
         "expsin": (("expsin", 0.5, (0.13, 0.27, 0.41)), O.k_expsin(0.5, (0.13, 0.27, 0.41))),
         "radial": (("radial", 2.99, 1.0, 0.45), O.k_radial())}


@pytest.mark.parametrize("case,L", [("tet", 0), ("tet", 1), ("tet", 4), ("shell", 0), ("shell", 1)])
@pytest.mark.parametrize("kind", sorted(SPECS))
@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_p2_matrix_free_apply(ctx, case, L, kind, dtype):
    coords, tets = M.tilted_tet() if case == "tet" else O.mesh_spherical_shell(2, 2, 0.55, 1.0)
    bl = "shell" if case == "shell" else None
    spec, kfun = SPECS[kind]
    op = O.P2DivKGrad(O.MacroMesh(coords, tets), L, L, kfun, blending=bl)
    pm = H.PrimitiveStorage.from_tets(coords, tets, ctx)
    A = H.P2ElementwiseBlendingDivKGradOperator(pm, L, L, ctx, k=spec, blending=bl)
    lev = op.levels[L]
    x = _rand(lev, 1)
    if dtype == "float32":
        x = x.astype(np.float32).astype(np.float64)
    fx, fy = (H.P2Function(n, pm, L, L, ctx, dtype) for n in "xy")
    fx.upload(L, x)
    A.apply(fx, fy, L, O.ALL)
    ref = op.apply(x, np.zeros_like(x), L, O.ALL)
    assert _relerr(fy.download(L), ref, lev.owned_mask(O.ALL)) < (1e-12 if dtype == "float64" else 4e-5)


@pytest.mark.parametrize("kind", sorted(SPECS))
def test_full_viscous_apply_smallest_level(ctx, kind):
    coords, tets = O.mesh_spherical_shell(2, 2, 0.55, 1.0)
    spec, kfun = SPECS[kind]
    op = O.P2FullViscous(O.MacroMesh(coords, tets), 0, 0, kfun, blending="shell")
    pm = H.PrimitiveStorage.from_tets(coords, tets, ctx)
    A = H.P2ElementwiseBlendingFullViscousOperator(pm, 0, 0, ctx, viscosity=spec, blending="shell")
    lev = op.levels[0]
    u = [_rand(lev, 10 + k) for k in range(3)]
    fu, fy = ([H.P2Function(n + str(k), pm, 0, 0, ctx) for k in range(3)] for n in "uy")
    for k in range(3):
        fu[k].upload(0, u[k])
    A.apply(fu, fy, 0, O.ALL)
    ref = op.apply(u, [np.zeros_like(v) for v in u], 0, O.ALL)
    for k in range(3):
        assert _relerr(fy[k].download(0), ref[k], lev.owned_mask(O.ALL)) < 1e-12


def _anchors_per_class(L):
    """The fewest micro-cell anchors (x, y, z), x + y + z < 2^L, of one coordinate parity."""
    n = 1 << L
    count = [0] * 8
    for z in range(n):
        for y in range(n - z):
            for x0 in (0, 1):
                count[(z & 1) * 4 + (y & 1) * 2 + x0] += len(range(x0, n - y - z, 2))
    return min(count)


def _full_blocks(cells, L):
    """Anchors per class on both sides of the change from the split pass to one anchor per thread, as the library
    counts them: the SMs with six blocks of 64 threads each."""
    import torch

    return cells * _anchors_per_class(L) >= torch.cuda.get_device_properties(0).multi_processor_count * 6 * 64


def test_p2_matrix_free_apply_full_blocks(ctx):
    """The one-anchor-per-thread pass against the stencil sweep of the constant operator (k = 1, no blending: the
    same matrix)."""
    coords, tets = M.cube_2x1x1()
    pm = H.PrimitiveStorage.from_tets(coords, tets, ctx)
    L = 6
    assert _full_blocks(len(tets), L)
    A = H.P2ElementwiseBlendingDivKGradOperator(pm, L, L, ctx, k=1.0)
    C = H.P2ConstantLaplaceOperator(pm, L, L, ctx)
    fx, fy, fz = (H.P2Function(n, pm, L, L, ctx) for n in "xyz")
    fx.fill_random(L, 7)
    A.apply(fx, fy, L, O.INNER)
    C.apply(fx, fz, L, O.INNER)
    y, z = fy.download(L), fz.download(L)
    assert np.abs(y - z).max() < 1e-12 * np.abs(z).max()


@pytest.mark.parametrize("nodal", [False, True])
@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_p2_full_blocks_on_the_shell(ctx, nodal, dtype):
    """The same pass with the shell map and a variable coefficient, closed form or node values, against the stored
    matrices of the same operator (FP64 sums of every pair; 1e-12 of the largest value, FP32 4e-5 as above)."""
    coords, tets = O.mesh_spherical_shell(5, 2, 0.55, 1.0)
    pm = H.PrimitiveStorage.from_tets(coords, tets, ctx)
    L = 4
    assert _full_blocks(len(tets), L) and not _full_blocks(len(tets), L - 1)
    kind = H.P2ElementwiseDivKGradOperator if nodal else H.P2ElementwiseBlendingDivKGradOperator
    spec = SPECS["expsin"][0]
    A, S = (kind(pm, L, L, ctx, k=spec, blending="shell") for _ in range(2))
    S.computeAndStoreLocalElementMatrices()
    fx, fy = (H.P2Function(n, pm, L, L, ctx, dtype) for n in "xy")
    gx, gy = (H.P2Function(n, pm, L, L, ctx) for n in ("gx", "gy"))
    fx.fill_random(L, 7)
    gx.upload(L, fx.download(L).astype(np.float64))
    A.apply(fx, fy, L, O.ALL)
    S.apply(gx, gy, L, O.ALL)
    y, z = fy.download(L), gy.download(L)
    assert np.abs(y - z).max() < (1e-12 if dtype == "float64" else 4e-5) * np.abs(z).max()


@pytest.mark.parametrize("case,L", [("shell", 2), ("shell", 4), ("box", 2), ("box", 4)])
@pytest.mark.parametrize("kind", ["const", "expsin"])
def test_fp32_passes_are_as_exact_as_their_type(ctx, case, L, kind):
    """FP32 results of the matrix-free operators against the same operators in FP64 on the same values: what a
    micro-cell computes once is computed in FP64 and rounded, so that a result carries the rounding of its
    terms, of the coefficient and of at most 24 partial sums: 2 unit roundoffs (1.2e-7) in the 2-norm."""
    coords, tets = O.mesh_spherical_shell(2, 2, 0.55, 1.0) if case == "shell" else M.cube_2x1x1()
    bl = "shell" if case == "shell" else None
    spec = SPECS[kind][0]
    pm = H.PrimitiveStorage.from_tets(coords, tets, ctx)
    out = {}
    start = {}
    for dtype in ("float32", "float64"):
        u, du = ([H.P2Function(n + str(k), pm, L, L, ctx, dtype) for k in range(3)] for n in ("u", "du"))
        p, dp = (H.P1Function(n, pm, L, L, ctx, dtype) for n in ("p", "dp"))
        for i, f in enumerate(u + [p]):
            if dtype == "float32":
                f.fill_random(L, 3 + i)
                start[i] = f.download(L)
            else:
                f.upload(L, start[i].astype(np.float64))
        A = H.P2ElementwiseBlendingDivKGradOperator(pm, L, L, ctx, k=spec, blending=bl)
        V = H.P2ElementwiseBlendingFullViscousOperator(pm, L, L, ctx, viscosity=spec, blending=bl)
        S = H.StokesUzawaMultigrid(ctx, pm, L, L, viscosity=spec, blending=bl)
        zero = [H.P2Function("z%d" % k, pm, L, L, ctx, dtype) for k in range(3)]
        zp = H.P1Function("zp", pm, L, L, ctx, dtype)

        def result(name, fns):
            out.setdefault(name, []).append(np.concatenate([f.download(L).astype(np.float64) for f in fns]))

        for f in zero + [zp] + du + [dp]:
            f.interpolate(0.0, L, H.All)
        A.apply(u[0], du[0], L, H.All)
        result("div k grad", du[:1])
        V.apply(u, du, L, H.All)
        result("full viscous", du)
        S.apply(zero, p, du, dp, L)
        result("divT", du)
        S.apply(u, zp, du, dp, L)
        result("div", [dp])
    for name, (low, ref) in out.items():
        assert np.linalg.norm(low - ref) <= 2 * 2.0**-24 * np.linalg.norm(ref), name


@pytest.mark.parametrize("case,L", [("tet", 0), ("tet", 1), ("tet", 4), ("shell", 0), ("shell", 2)])
@pytest.mark.parametrize("dtype", ["float64", "float32", "float16"])
def test_p2_stored_apply(ctx, case, L, dtype):
    """Stored matrices at the levels without inner nodes, with segments shorter than a block and with
    several macro-cells in one block; FP32 sums up to 65 rounded products per macro-cell: 100 eps; FP16 holds the
    vectors only, so its result differs by their rounding, half of 2^-10, and that of the FP32 sum."""
    coords, tets = M.tilted_tet() if case == "tet" else O.mesh_spherical_shell(2, 2, 0.55, 1.0)
    bl = "shell" if case == "shell" else None
    spec, kfun = SPECS["expsin"]
    op = O.P2DivKGrad(O.MacroMesh(coords, tets), L, L, kfun, blending=bl)
    pm = H.PrimitiveStorage.from_tets(coords, tets, ctx)
    A = H.P2ElementwiseBlendingDivKGradOperator(pm, L, L, ctx, k=spec, blending=bl)
    A.computeAndStoreLocalElementMatrices()
    lev = op.levels[L]
    x = _rand(lev, 1)
    x = x.astype(dtype).astype(np.float64)
    fx, fy = (H.P2Function(n, pm, L, L, ctx, dtype) for n in "xy")
    fx.upload(L, x)
    for flag in (O.INNER, O.ALL):
        fy.interpolate(0.0, L, H.All)
        A.apply(fx, fy, L, flag)
        ref = op.apply(x, np.zeros_like(x), L, flag)
        err = np.abs(fy.download(L).astype(np.float64) - ref)[lev.owned_mask(O.ALL)].max()
        tol = {"float64": 1e-12, "float32": 1.2e-5, "float16": 2.0**-11 + 1.2e-5}[dtype]
        assert err <= tol * max(np.abs(ref).max(), 1e-300)


def test_fp32_stored_weights_in_slabs(ctx):
    """FP32 weights of a level whose FP64 weights (2.5 GB) do not fit beside them (1.3 GB): built from slabs of
    macro-cells, with the same bits as weights rounded from all FP64 ones at once."""
    import torch

    coords, tets = O.mesh_spherical_shell(3, 2, 0.55, 1.0)
    pm = H.PrimitiveStorage.from_tets(coords, tets, ctx)
    L = 5
    fx, fy = (H.P2Function(n, pm, L, L, ctx, "float32") for n in "xy")
    fx.fill_random(L, 1)

    def operator():
        A = H.P2ElementwiseBlendingDivKGradOperator(pm, L, L, ctx, k=SPECS["expsin"][0], blending="shell")
        A.computeAndStoreLocalElementMatrices()
        return A

    A = operator()
    ctx.synchronize()
    torch.cuda.empty_cache()
    room = int(2.4e9)
    filler = [torch.empty(max(torch.cuda.mem_get_info()[0] - room, 1), dtype=torch.uint8, device="cuda")]
    assert torch.cuda.mem_get_info()[0] < 1.1 * room
    A.apply(fx, fy, L, H.All)
    low = fy.download(L)
    filler.clear()
    torch.cuda.empty_cache()
    B = operator()
    dx, dy = (H.P2Function(n, pm, L, L, ctx) for n in ("dx", "dy"))
    dx.upload(L, fx.download(L).astype(np.float64))
    B.apply(dx, dy, L, H.All)
    fy.interpolate(0.0, L, H.All)
    B.apply(fx, fy, L, H.All)
    np.testing.assert_array_equal(fy.download(L), low)
    ref = dy.download(L)
    assert np.abs(low - ref).max() <= 1.2e-5 * np.abs(ref).max()
