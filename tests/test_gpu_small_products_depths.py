"""The FP32 translations' 32 x 32 tiles where they are chosen: depths that are
multiples of four but not of the 32-deep step, and ragged rows.  One right-hand
side takes the small tiles, 96 take the large ones: each against the direct sum
and both against each other (same split and order of the depth, atomic sums in
any order).

Tolerances: the expansions at 76 to 148 surface points and MAC 0.3 reach 1e-5
for the single layer: 2e-5; two orders of atomic FP32 sums agree to 1e-6."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [76, 100, 148])
@pytest.mark.parametrize("path", [1, 4])
def test_small_and_large_tiles(order, path):
    from tbempy import ThreeD, meshes
    locs, nrm, w = meshes.sphere_points(2)
    locs, nrm, w = locs[:931], nrm[:931], w[:931]
    K = ThreeD.LaplaceSingle()
    op = ThreeD.FMMOperator(K, locs, nrm, locs, nrm, w, ThreeD.FMMConfig(0.3, order, 17, 0.05, False),
                            precision="mixed", m2l_path=path)
    rng = np.random.default_rng(order)
    x = rng.uniform(-1, 1, (96, len(locs)))
    z = rng.uniform(-1, 1, (96, len(locs)))
    many, many_t = op.apply(x), op.apply_adjoint(z)
    for r in (0, 41, 95):
        for got, rest, ref in (
                (op.apply(x[r]), many[r], oracle.direct("LaplaceSingle", locs, nrm, locs, nrm, w, x[r])),
                # A = K W with K symmetric: A^T z = W K z
                (op.apply_adjoint(z[r]), many_t[r],
                 w * oracle.direct("LaplaceSingle", locs, nrm, locs, nrm, np.ones_like(w), z[r]))):
            assert np.linalg.norm(got - ref) < 2e-5 * np.linalg.norm(ref)
            assert np.linalg.norm(rest - ref) < 2e-5 * np.linalg.norm(ref)
            assert np.linalg.norm(got - rest) < 1e-6 * np.linalg.norm(ref)
