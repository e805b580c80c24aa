"""The plain form's FP64 translations (one-warp tiles of 8 rows x 4 to 16
columns) where their tiles have remainders: surfaces whose row counts are one
below, at and above a multiple of 8, from one to seven right-hand sides, and
trees from a single leaf to several levels.

Tolerance 1e-10 against the oracle with its pseudo-inverses installed: the bar
of the plain form at surfaces of a few dozen points, where the reference's own
one-ulp floor is below 1e-12.  Each right-hand side of a multi-RHS apply adds
in the order of a single apply.
"""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("kernel,order", [("LaplaceSingle", 15), ("LaplaceSingle", 16), ("LaplaceSingle", 33),
                                          ("ElasticDisplacement", 8), ("ElasticDisplacement", 19)])
@pytest.mark.parametrize("n_points,leaf", [(30, 40), (700, 12)])
@pytest.mark.parametrize("n_rhs", [1, 3, 7])
def test_plain_translations_at_tile_edges(kernel, order, n_points, leaf, n_rhs):
    from tbempy import ThreeD
    rng = np.random.default_rng(11)
    locs = rng.uniform(-1, 1, (n_points, 3))
    nrm = rng.normal(size=(n_points, 3))
    nrm /= np.linalg.norm(nrm, axis=1)[:, None]
    w = rng.uniform(0.5, 1.0, n_points)
    orc = oracle.OracleFMM(kernel, locs, nrm, locs, nrm, w, 0.3, order, leaf, 0.05, False)
    K = getattr(ThreeD, kernel)
    op = ThreeD.FMMOperator(K(1.0, 0.25) if kernel.startswith("Elastic") else K(), locs, nrm, locs, nrm, w,
                            ThreeD.FMMConfig(0.3, order, leaf, 0.05, False))
    for which in (0, 1):
        for lev in range(op.n_c2e_levels(which)):
            op.set_c2e(which, lev, orc.c2e[which][lev])
    x = rng.uniform(-1, 1, (n_rhs, op.n_cols()))
    y = op.apply(x)
    z = rng.uniform(-1, 1, (n_rhs, op.n_rows()))
    wz = op.apply_adjoint(z)
    for r in range(n_rhs):
        assert rel(y[r], orc.apply(x[r])) < 1e-10
        a, b = float(z[r] @ y[r]), float(wz[r] @ x[r])
        assert abs(a - b) < 1e-10 * np.linalg.norm(z[r]) * np.linalg.norm(y[r])
