"""The precision form's applies, forward and transposed, entry by entry against
FP64 direct sums that share nothing with the operators: the direct operator and
the density gradient of the direct gradient pass (A^T r).  Operators on one
surface and on two (most M2L classes then have one to four pairs, with kernels
of their own for one right-hand side), for one and five right-hand sides.

Tolerance: the expansions of order 152 (Laplace) and 296 at MAC 0.3 with FP32
products reach 1e-6 of the norm, 2e-6 is asserted; an entry is within 3e-5 of
the larger of itself and the rms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def points(surface, size, n_obs):
    from tbempy import meshes
    if surface == "sphere":
        src, nrm, w = meshes.sphere_points(size)
        return src, nrm, src, nrm, w
    v, t, _ = meshes.dipping_fault(size, 45.0)
    v = v.copy()
    v[:, 2] += 0.05 * np.sin(3 * v[:, 0]) * np.cos(2 * v[:, 1])
    src, nrm, w = meshes.points_from_mesh(v, t)
    rng = np.random.default_rng(17)
    obs = np.ascontiguousarray(np.concatenate([rng.uniform(-3, 3, (n_obs, 2)), np.zeros((n_obs, 1))], axis=1))
    return obs, np.tile([0.0, 0.0, 1.0], (n_obs, 1)), src, nrm, w


@pytest.mark.parametrize("kernel,order,surface,size,n_obs", [
    ("LaplaceSingle", 152, "sphere", 3, 0), ("LaplaceDouble", 152, "sphere", 3, 0),
    ("ElasticDisplacement", 296, "sphere", 3, 0), ("ElasticTraction", 296, "sphere", 3, 0),
    ("ElasticDisplacement", 296, "fault", 27, 1777), ("LaplaceSingle", 296, "fault", 30, 2500)])
@pytest.mark.parametrize("path", [0, 5])
def test_entries_against_direct_sums(kernel, order, surface, size, n_obs, path):
    from tbempy import ThreeD
    ol, on, sl, sn, w = points(surface, size, n_obs)
    K = getattr(ThreeD, kernel)
    K = K(1.0, 0.25) if kernel.startswith("Elastic") else K()
    op = ThreeD.FMMOperator(K, ol, on, sl, sn, w, ThreeD.FMMConfig(0.3, order, 64, 0.05, False), precision="mixed",
                            m2l_path=path)
    assert op.m2l_ranks()[0] > 0
    rng = np.random.default_rng(31)
    direct = ThreeD.DirectOperator(K, ol, on, sl, sn, w)
    for n_rhs in (1, 5):
        x = rng.uniform(-1, 1, (n_rhs, op.n_cols()))
        z = rng.uniform(-1, 1, (n_rhs, op.n_rows()))
        y, v = op.apply(x), op.apply_adjoint(z)
        for r in {0, n_rhs - 1}:
            for got, ref in ((y[r], direct.apply(x[r])),
                             (v[r], ThreeD.direct_gradients(K, ol, on, sl, sn, w, x[r], z[r])["x"])):
                assert np.linalg.norm(got - ref) <= 2e-6 * np.linalg.norm(ref)
                assert np.all(np.abs(got - ref) <= 3e-5 * np.maximum(np.abs(ref), np.sqrt(np.mean(ref * ref))))
