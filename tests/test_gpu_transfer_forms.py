"""Linear transfers on both sides of the change from listed points to rows (64 points per macro-edge), with
edges and vertices of many cells, one-cell (Neumann) faces, both update types: against the oracle's
matrices up to level 4 (1e-12, as the other transfer tests), and for the large levels by R = P^T."""

import numpy as np
import pytest

import hyteg_b200 as H
from oracle import hyteg_oracle as O
from tests import meshes as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh", ["unit_tet", "pyramid_4", "octahedron_8", "cube_2x1x1"])
@pytest.mark.parametrize("L", [1, 2, 4])
@pytest.mark.parametrize("neumann", [False, True])
def test_transfers_match_oracle(ctx, mesh, L, neumann):
    coords, tets = M.ALL[mesh]()
    om = O.MacroMesh(coords, tets, bc_types={0: O.INNER, 1: O.NEUMANN} if neumann else None)
    op = O.P1ConstantLaplace(om, L - 1, L)
    tr = O.Transfer(op)
    pm = H.PrimitiveStorage.from_tets(coords, tets, ctx)
    if neumann:
        pm.set_bc_type(1, H.NeumannBoundary)
    flag = H.Inner | H.NeumannBoundary
    rng = np.random.default_rng(L)
    vec = {}
    for l in (L - 1, L):
        lev = op.levels[l]
        v = np.zeros(lev.size)
        v[lev.owned] = rng.uniform(-1, 1, lev.owned.size)
        vec[l] = lev.sync(v)
    f = H.P1Function("f", pm, L - 1, L, ctx)

    def check(l, ref):
        own = op.levels[l].owned_mask(O.ALL)
        got = f.download(l)
        assert np.abs(got[own] - ref[own]).max() <= 1e-12 * max(np.abs(ref[own]).max(), 1e-300)
        d, s = op.levels[l].copy_map()
        np.testing.assert_array_equal(got[d], got[s])

    for l in vec:
        f.upload(l, vec[l])
    H.P1toP1LinearRestriction().restrict(f, L, flag)
    check(L - 1, tr.restrict(vec[L], vec[L - 1].copy(), L, flag))
    for add in (True, False):
        for l in vec:
            f.upload(l, vec[l])
        P = H.P1toP1LinearProlongation()
        (P.prolongateAndAdd if add else P.prolongate)(f, L - 1, flag)
        check(L, tr.prolongate(vec[L - 1], vec[L].copy(), L, flag, add=add))


@pytest.mark.parametrize("L", [6, 7, 8])
def test_restriction_is_the_transpose(ctx, L):
    coords, tets = M.cube_6()
    pm = H.PrimitiveStorage.from_tets(coords, tets, ctx)
    a, b = (H.P1Function(n, pm, L - 1, L, ctx) for n in "ab")
    a.fill_random(L, 1)
    b.fill_random(L - 1, 2)
    for f, l in ((a, L), (b, L - 1)):
        f.interpolate(0.0, l, H.DirichletBoundary)
    H.P1toP1LinearRestriction().restrict(a, L, H.Inner)
    H.P1toP1LinearProlongation().prolongate(b, L - 1, H.Inner)
    left, right = a.dotGlobal(b, L - 1, H.Inner), a.dotGlobal(b, L, H.Inner)
    # both sums have up to 1.7e7 terms of size one: rounding grows like their square root
    assert abs(left - right) <= 1e-12 * np.sqrt(a.dotGlobal(a, L, H.Inner) * b.dotGlobal(b, L, H.Inner))


@pytest.mark.parametrize("L", [4, 7])
@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_prolongation_of_large_values(ctx, L, dtype):
    """Values above half of the largest number interpolate to themselves: copied at coarse nodes, and the halves
    summed at the others."""
    coords, tets = M.cube_6()
    pm = H.PrimitiveStorage.from_tets(coords, tets, ctx)
    f = H.P1Function("f", pm, L - 1, L, ctx, dtype)
    got = {}
    for value in (1.0, 0.9 * float(np.finfo(dtype).max)):
        f.upload(L - 1, np.full(f.download(L - 1).shape, value, dtype=dtype))
        f.upload(L, np.zeros(f.download(L).shape, dtype=dtype))
        H.P1toP1LinearProlongation().prolongate(f, L - 1, H.All)
        got[value] = f.download(L)
    ones, big = got.values()
    np.testing.assert_array_equal(big, np.where(ones == 1.0, np.asarray(value, dtype=dtype), np.asarray(0.0, dtype=dtype)))
    assert np.count_nonzero(ones) > (2 ** L - 1) ** 3
