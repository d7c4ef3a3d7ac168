"""P2 constant stencils on both sides of the change from one thread per node to the tiled sweep, on meshes
with edges and vertices of many cells and with one-cell (Neumann) faces: against the oracle on small levels
and the elementwise operator with k = 1 on large ones (the same matrix; 1e-12 of the largest value)."""

import numpy as np
import pytest

import hyteg_b200 as H
from oracle import hyteg_oracle as O
from tests import meshes as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh", ["unit_tet", "pyramid_4", "octahedron_8"])
@pytest.mark.parametrize("L", [0, 1, 3])
@pytest.mark.parametrize("neumann", [False, True])
def test_p2_constant_matches_oracle(ctx, mesh, L, neumann):
    coords, tets = M.ALL[mesh]()
    om = O.MacroMesh(coords, tets, bc_types={0: O.INNER, 1: O.NEUMANN} if neumann else None)
    op = O.P2DivKGrad(om, L, L, lambda P: np.ones(np.asarray(P).shape[:-1]))
    lev = op.levels[L]
    pm = H.PrimitiveStorage.from_tets(coords, tets, ctx)
    if neumann:
        pm.set_bc_type(1, H.NeumannBoundary)
    A = H.P2ConstantLaplaceOperator(pm, L, L, ctx)
    flag = H.Inner | H.NeumannBoundary
    rng = np.random.default_rng(L)
    vec = {}
    for n in ("x", "b", "y"):
        v = np.zeros(lev.size)
        v[lev.owned] = rng.uniform(-1, 1, lev.owned.size)
        vec[n] = lev.sync(v)
    f = {n: H.P2Function(n, pm, L, L, ctx) for n in vec}
    for n in vec:
        f[n].upload(L, vec[n])
    own = lev.owned_mask(O.ALL)

    def check(ref):
        got = f["y"].download(L)
        assert np.abs(got[own] - ref[own]).max() <= 1e-12 * max(np.abs(ref[own]).max(), 1e-300)
        d, s = lev.copy_map()
        np.testing.assert_array_equal(got[d], got[s])

    for flag_ in (flag, O.ALL):
        f["y"].upload(L, vec["y"])
        A.apply(f["x"], f["y"], L, flag_)
        ref = op.apply(vec["x"], vec["y"].copy(), L, flag_)
        check(ref)
    A.smooth_jac(f["y"], f["b"], f["x"], 0.6, L, flag)
    check(op.smooth_jac(ref.copy(), vec["b"], vec["x"], 0.6, L, flag))


@pytest.mark.parametrize("cells,L", [(6, 5), (6, 6), (6, 7), (60, 5), (120, 5), (120, 4)])
@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_p2_constant_equals_elementwise(ctx, cells, L, dtype):
    """Both sides of the changes of kernel: 64 and 128 nodes per edge, and 2.4 and 4.8 million nodes at 64.  FP32: 65
    products of values up to one and weights of either sign, 100 eps."""
    coords, tets = M.cube_6() if cells == 6 else O.mesh_spherical_shell(2, 1 + cells // 60, 0.55, 1.0)
    pm = H.PrimitiveStorage.from_tets(coords, tets, ctx)
    C = H.P2ConstantLaplaceOperator(pm, L, L, ctx)
    A = H.P2ElementwiseBlendingDivKGradOperator(pm, L, L, ctx, k=1.0)
    fx, fy, fz = (H.P2Function(n, pm, L, L, ctx, dtype) for n in "xyz")
    fx.fill_random(L, 7)
    A.apply(fx, fy, L, O.INNER)
    C.apply(fx, fz, L, O.INNER)
    y, z = fy.download(L), fz.download(L)
    assert np.abs(y - z).max() < (1e-12 if dtype == "float64" else 1.2e-5) * np.abs(y).max()
