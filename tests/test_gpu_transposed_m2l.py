"""The transposed apply of the precision form (the M2L operators taken
transposed from the same tensor-core planes; the transposed leaf operators) at
ranks that leave its 128-row and 64-deep tiles with remainders, for every tile
shape, against the forward apply: <z, A x> = <A^T z, x>.

Tolerance: both sides run in FP32 with FP32-accurate products and compensated
near-field sums (1e-7 of the result's norm); 2e-6 of |z| |A x| leaves room for
the norms' ratio."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel,order", [("LaplaceSingle", 152), ("LaplaceDouble", 152),
                                          ("ElasticDisplacement", 296), ("ElasticTraction", 296)])
@pytest.mark.parametrize("shape", [1, 2, 3, 4])
@pytest.mark.parametrize("n_rhs", [1, 5])
def test_transposed_apply_is_the_transpose(kernel, order, shape, n_rhs):
    from tbempy import ThreeD, meshes
    locs, nrm, w = meshes.sphere_points(3)
    K = getattr(ThreeD, kernel)
    op = ThreeD.FMMOperator(K(1.0, 0.25) if kernel.startswith("Elastic") else K(), locs, nrm, locs, nrm, w,
                            ThreeD.FMMConfig(0.3, order, 30, 0.05, False), precision="mixed", m2l_path=5,
                            tc_shape=shape)
    assert op.m2l_ranks()[0] > 0
    rng = np.random.default_rng(9)
    x = rng.uniform(-1, 1, (n_rhs, op.n_cols()))
    z = rng.uniform(-1, 1, (n_rhs, op.n_rows()))
    y, v = op.apply(x), op.apply_adjoint(z)
    for r in range(n_rhs):
        assert abs(float(z[r] @ y[r]) - float(v[r] @ x[r])) < 2e-6 * np.linalg.norm(z[r]) * np.linalg.norm(y[r])
