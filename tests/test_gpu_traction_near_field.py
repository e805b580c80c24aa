"""The FP64 near field of the traction kernels (three multiply-adds per
component), entry by entry: operators whose points are one leaf, applied to
every unit vector, forward and transposed, in 3D and 2D, against the oracle's
direct sum.

Tolerance: an entry is about 60 FP64 operations on terms no larger than its
block's largest entry, and the separations are differences of rounded
coordinates (2^-53 over the smallest separation, 1/100 here): 1e-11 of the
block's largest entry."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [3, 2])
@pytest.mark.parametrize("kernel", ["ElasticTraction", "ElasticAdjointTraction"])
@pytest.mark.parametrize("n_obs,n_src", [(37, 29), (29, 37), (3, 41)])
def test_every_entry(dim, kernel, n_obs, n_src):
    from tbempy import ThreeD, TwoD
    rng = np.random.default_rng(n_obs)

    def grid(n, shift):  # jittered grid: separations of at least 1/100
        m = int(np.ceil(n ** (1 / dim)))
        p = np.stack(np.meshgrid(*[np.arange(m)] * dim, indexing="ij"), axis=-1).reshape(-1, dim)[:n]
        p = (p + 0.3 * rng.uniform(-1, 1, p.shape)) / m + shift
        q = rng.normal(size=p.shape)
        return np.ascontiguousarray(p), q / np.linalg.norm(q, axis=1)[:, None]

    (ol, on), (sl, sn) = grid(n_obs, 0.0), grid(n_src, 0.013)
    w = rng.uniform(0.5, 1.0, n_src)
    d = np.linalg.norm(ol[:, None] - sl[None], axis=2)
    keep = d.min(axis=1) > 0.01
    ol, on, n_obs = np.ascontiguousarray(ol[keep]), np.ascontiguousarray(on[keep]), int(keep.sum())
    K = getattr(TwoD if dim == 2 else ThreeD, kernel)(1.0, 0.25)
    op = ThreeD.FMMOperator(K, ol, on, sl, sn, w, ThreeD.FMMConfig(0.3, 16, 64, 0.05, False))
    A = np.stack([oracle.direct(kernel, ol, on, sl, sn, w, e) for e in np.eye(dim * n_src)], axis=1)
    scale = np.abs(A).reshape(dim, n_obs, dim, n_src).max(axis=(0, 2))
    tol = 1e-11 * np.tile(scale, (dim, dim))
    assert np.all(np.abs(op.apply(np.eye(dim * n_src)).T - A) <= tol)
    assert np.all(np.abs(op.apply_adjoint(np.eye(dim * n_obs)) - A) <= tol)
    direct = ThreeD.DirectOperator(K, ol, on, sl, sn, w) if dim == 3 else None
    if direct:
        assert np.all(np.abs(direct.apply(np.eye(dim * n_src)).T - A) <= tol)
