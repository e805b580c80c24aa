"""The FP64 compressed form's M2L through digit planes entry by entry against
the same operator on the FP64 pipe (m2l_path 4): rank tolerances down to 1e-12,
where the compressed coefficients reach furthest down the singular values, and
densities over twelve decades.  Digits are cut relative to the largest entry of
a row and a column; coefficients graded against the operators would show here.

Tolerance: the digits hold 2^-58 of the largest products of a row and a column
and the FP64 pipe rounds at 2^-53 per addition, both over sums of at most 704
terms; 1e-13 of the larger of an entry and the result's rms leaves a factor of
ten for coefficients larger than the result.  Infinities and NaNs come out in
the same places on both paths."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel,tol", [("LaplaceDouble", 1e-9), ("LaplaceDouble", 1e-12), ("LaplaceSingle", 1e-9),
                                        ("ElasticDisplacement", 1e-7), ("ElasticDisplacement", 1e-9),
                                        ("ElasticDisplacement", 1e-12), ("ElasticTraction", 1e-12)])
def test_digit_planes_entry_by_entry(kernel, tol):
    from tbempy import ThreeD, meshes
    locs, nrm, w = meshes.sphere_points(3)
    K = getattr(ThreeD, kernel)
    K = K(1.0, 0.25) if kernel.startswith("Elastic") else K()
    ops = [ThreeD.FMMOperator(K, locs, nrm, locs, nrm, w, ThreeD.FMMConfig(0.3, 296, 30, 0.05, False),
                              precision="fp64_compressed", m2l_path=p, m2l_rank_tol=tol) for p in (0, 4)]
    rng = np.random.default_rng(12)
    for decades in (0, 6, 12):
        x = rng.uniform(-1, 1, ops[0].n_cols()) * 10.0 ** rng.uniform(-decades, 0, ops[0].n_cols())
        y, ref = (op.apply(x) for op in ops)
        assert ops[0].last_launches() == ops[1].last_launches() + 1  # the planes are in use
        assert np.all(np.abs(y - ref) <= 1e-13 * np.maximum(np.abs(ref), np.sqrt(np.mean(ref * ref))))
    for bad in (np.inf, -np.inf, np.nan):
        x = rng.uniform(-1, 1, ops[0].n_cols())
        x[29] = bad
        y, ref = (op.apply(x) for op in ops)
        assert np.array_equal(np.isnan(y), np.isnan(ref))
        assert np.array_equal(y[np.isinf(ref)], ref[np.isinf(ref)])
