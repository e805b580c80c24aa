"""The precision form's FP32 translations in launches of few columns (32 x 32
tiles) at row, column and depth remainders, forward and transposed, against the
direct sum.

The paths are the FP32 ones (m2l_path 1: uncompressed, 4: compressed).
Tolerance 2e-5: the expansions at 152 surface points and MAC 0.3 reach 1e-6, at
99 and 75 points 1e-5 for the single layer; <z, A x> = <A^T z, x> holds to FP32
rounding, 1e-5 of |z| |A x|."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [75, 99, 152])
@pytest.mark.parametrize("path", [1, 4])
@pytest.mark.parametrize("n_rhs", [1, 3, 7])
def test_small_products(order, path, n_rhs):
    from tbempy import ThreeD, meshes
    locs, nrm, w = meshes.sphere_points(2)
    locs, nrm, w = locs[:931], nrm[:931], w[:931]
    K = ThreeD.LaplaceSingle()
    op = ThreeD.FMMOperator(K, locs, nrm, locs, nrm, w, ThreeD.FMMConfig(0.3, order, 17, 0.05, False),
                            precision="mixed", m2l_path=path)
    rng = np.random.default_rng(order)
    x = rng.uniform(-1, 1, (n_rhs, len(locs)))
    z = rng.uniform(-1, 1, (n_rhs, len(locs)))
    y, v = op.apply(x), op.apply_adjoint(z)
    for r in range(n_rhs):
        ref = oracle.direct("LaplaceSingle", locs, nrm, locs, nrm, w, x[r])
        assert np.linalg.norm(y[r] - ref) < 2e-5 * np.linalg.norm(ref)
        assert abs(float(z[r] @ y[r]) - float(v[r] @ x[r])) < 1e-5 * np.linalg.norm(z[r]) * np.linalg.norm(y[r])
