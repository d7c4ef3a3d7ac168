"""P1 operators with stored matrices (eight weights per slot, the other seven directions read from the
neighbours): every operation's epilogue at levels without inner points, with cells shorter than a block and
with several blocks per cell, against the matrix-free operator.  FP64: 15 products per cell, summed in
another order, 1e-13 of the largest value (as the stored-matrix tests elsewhere); FP32: 15 products per cell
and up to 30 cells, 64 eps; FP16 vectors: both results rounded to half of 2^-10 as well."""

import numpy as np
import pytest

import hyteg_b200 as H
from oracle import hyteg_oracle as O
from tests import meshes as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case,L", [("tet", 0), ("tet", 1), ("tet", 5), ("shell", 0), ("shell", 3)])
@pytest.mark.parametrize("dtype", ["float64", "float32", "float16"])
def test_p1_stored_equals_matrix_free(ctx, case, L, dtype):
    coords, tets = M.tilted_tet() if case == "tet" else O.mesh_spherical_shell(2, 3, 0.55, 1.0)
    bl = "shell" if case == "shell" else None
    pm = H.PrimitiveStorage.from_tets(coords, tets, ctx)
    k = ("expsin", 0.5, (0.13, 0.27, 0.41))
    A, S = (H.P1ElementwiseBlendingDivKGradOperator(pm, L, L, ctx, k=k, blending=bl) for _ in range(2))
    S.computeAndStoreLocalElementMatrices()
    f = {n: H.P1Function(n, pm, L, L, ctx, dtype) for n in ("x", "b", "y", "z")}
    f["x"].fill_random(L, 3)
    f["b"].fill_random(L, 4)
    tol = {"float64": 1e-13, "float32": 8e-6, "float16": 2.0**-10 + 8e-6}[dtype]
    for flag in (O.INNER, O.ALL):
        for op in ("apply", "add", "jacobi"):
            for A_, out in ((A, "y"), (S, "z")):
                f[out].fill_random(L, 5)
                if op == "jacobi":
                    A_.smooth_jac(f[out], f["b"], f["x"], 0.6, L, flag)
                else:
                    A_.apply(f["x"], f[out], L, flag, H.Add if op == "add" else H.Replace)
            y, z = f["y"].download(L), f["z"].download(L)
            assert np.abs(y - z).max() <= tol * np.abs(y).max(), (flag, op)
