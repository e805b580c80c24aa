"""M2L groups of a few pairs (FP32 products from memory): observers on a surface
over a warped fault, where most (level difference, offset) classes have one to
four pairs, against the same operator with every group on the tensor cores
(m2l_path=5), forward and transposed, for one right-hand side (the small groups
leave the tensor cores) and three (they do not).

Tolerance: both take FP32 operators and FP32 sums of at most 296 products, on
the tensor cores from three bf16 terms (2^-22 of a product): 2e-6 of the
result's largest value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel,size,n_obs,tol", [
    ("ElasticDisplacement", 32, 4096, 1e-7), ("ElasticDisplacement", 27, 1777, 1e-7), ("ElasticTraction", 30, 2500, 1e-7),
    ("LaplaceSingle", 32, 4096, 1e-7),  # ranks below 128
    ("ElasticDisplacement", 24, 1500, 1e-8)])  # larger ranks: more pieces of a row per lane
def test_small_groups_match_the_tensor_cores(kernel, size, n_obs, tol):
    from tbempy import ThreeD, meshes
    v, t, _ = meshes.dipping_fault(size, 45.0)
    v = v.copy()
    v[:, 2] += 0.05 * np.sin(3 * v[:, 0]) * np.cos(2 * v[:, 1])
    src, nrm, w = meshes.points_from_mesh(v, t)
    rng = np.random.default_rng(17)
    obs = np.ascontiguousarray(np.concatenate([rng.uniform(-3, 3, (n_obs, 2)), np.zeros((n_obs, 1))], axis=1))
    onrm = np.tile([0.0, 0.0, 1.0], (n_obs, 1))
    K = getattr(ThreeD, kernel)
    k = K(1.0, 0.25) if kernel.startswith("Elastic") else K()
    ops = [ThreeD.FMMOperator(k, obs, onrm, src, nrm, w, ThreeD.FMMConfig(0.3, 296, 64, 0.05, False),
                              precision="mixed", m2l_path=p, m2l_rank_tol=tol) for p in (0, 5)]
    for n_rhs in (1, 3):
        x = rng.uniform(-1, 1, (n_rhs, ops[0].n_cols()))
        z = rng.uniform(-1, 1, (n_rhs, ops[0].n_rows()))
        y, v_ = ([np.asarray(op.apply(x)) for op in ops], [np.asarray(op.apply_adjoint(z)) for op in ops])
        if n_rhs == 1:  # the small groups have a launch of their own
            assert ops[0].last_launches() != ops[1].last_launches()
        for a, b in (y, v_):
            assert np.abs(a - b).max() < 2e-6 * np.abs(b).max()
