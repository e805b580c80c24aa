"""The FP64 compressed form's M2L through digit planes on the tensor cores,
against the same operator on the FP64 pipe (m2l_path 4), at ranks and group
sizes that leave its 128 x 64 tiles and 32-deep chunks with remainders.

Tolerance: the split is error free up to 2^-56 of each row's and column's
largest entry and the FP64 pipe rounds at 2^-53 per addition, so the two differ
by a few rounding errors of a sum of a few hundred terms: 1e-13 of the norm.
Powers of two scale both without a rounding: results scale exactly up to the
order of the atomic sums (1e-13 again)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("kernel,order,sub,leaf", [("LaplaceSingle", 152, 3, 30), ("LaplaceDouble", 296, 3, 40),
                                                   ("ElasticDisplacement", 296, 3, 30), ("LaplaceSingle", 296, 4, 25)])
@pytest.mark.parametrize("n_rhs", [1, 3])
def test_digit_planes_match_the_fp64_pipe(kernel, order, sub, leaf, n_rhs):
    from tbempy import ThreeD, meshes
    locs, nrm, w = meshes.sphere_points(sub)
    K = getattr(ThreeD, kernel)
    K = K(1.0, 0.25) if kernel.startswith("Elastic") else K()
    cfg = ThreeD.FMMConfig(0.3, order, leaf, 0.05, False)
    ops = [ThreeD.FMMOperator(K, locs, nrm, locs, nrm, w, cfg, precision="fp64_compressed", m2l_path=p)
           for p in (0, 4)]
    rng = np.random.default_rng(2)
    x = rng.uniform(-1, 1, (n_rhs, ops[0].n_cols())) * 10.0 ** rng.uniform(-6, 0, (n_rhs, ops[0].n_cols()))
    y, ref = ops[0].apply(x), ops[1].apply(x)
    for r in range(n_rhs):
        assert rel(y[r], ref[r]) < 1e-13
    for p in (-700, 600):
        assert rel(np.ldexp(ops[0].apply(np.ldexp(x, p)), -p), y) < 1e-13
    assert not ops[0].apply(np.zeros_like(x)).any()


def test_a_not_finite_density_reaches_the_result():
    from tbempy import ThreeD, meshes
    locs, nrm, w = meshes.sphere_points(3)
    op = ThreeD.FMMOperator(ThreeD.LaplaceSingle(), locs, nrm, locs, nrm, w,
                            ThreeD.FMMConfig(0.3, 152, 30, 0.05, False), precision="fp64_compressed")
    x = np.ones(len(locs))
    x[17] = np.inf
    assert not np.isfinite(op.apply(x)).all()
    x[17] = np.nan
    assert np.isnan(op.apply(x)).any()
    x[17] = 1.0
    assert np.isfinite(op.apply(x)).all()
