"""Near fields whose source lists differ by orders of magnitude (a dense cluster
beside scattered points: a few leaves see almost every point), where the FP64
passes give long lists a warp or a whole CTA per target, against the direct sum;
and the direct sum itself on both sides of its threads-per-target rule.

Tolerances: with the same pairs in the near field the forms differ from the
direct sum by their expansions (order 152, MAC 0.3: below 1e-6); two direct
sums of n terms of either sign in FP64 differ by less than n 2^-53 of the sum
of magnitudes, 1e-11 here."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


def clustered(n, seed):
    rng = np.random.default_rng(seed)
    a = rng.uniform(-1, 1, (n // 20, 3))
    b = 0.02 * rng.normal(size=(n - len(a), 3)) + [0.3, 0.2, -0.1]
    locs = np.concatenate([a, b])
    nrm = rng.normal(size=locs.shape)
    return locs, nrm / np.linalg.norm(nrm, axis=1)[:, None], rng.uniform(0.5, 1.0, len(locs))


@pytest.mark.parametrize("precision", ["fp64", "fp64_compressed"])
@pytest.mark.parametrize("n_rhs", [1, 3])
def test_long_lists_match_the_direct_sum(precision, n_rhs):
    from tbempy import ThreeD
    locs, nrm, w = clustered(9001, 5)
    K = ThreeD.LaplaceSingle()
    op = ThreeD.FMMOperator(K, locs, nrm, locs, nrm, w, ThreeD.FMMConfig(0.3, 152, 60, 0.05, False),
                            precision=precision)
    x = np.random.default_rng(6).uniform(-1, 1, (n_rhs, len(locs)))
    y, v = op.apply(x), op.apply_adjoint(x)
    for r in range(n_rhs):
        ref = oracle.direct("LaplaceSingle", locs, nrm, locs, nrm, w, x[r])
        assert np.linalg.norm(y[r] - ref) < 1e-6 * np.linalg.norm(ref)
        # A = K W with K symmetric: A^T x = W K x
        ref_t = w * oracle.direct("LaplaceSingle", locs, nrm, locs, nrm, np.ones_like(w), x[r])
        assert np.linalg.norm(v[r] - ref_t) < 1e-6 * np.linalg.norm(ref_t)


@pytest.mark.parametrize("n_obs", [1, 5, 127, 1025, 38911, 38912])
def test_direct_sum_at_the_threads_per_target_rule(n_obs):
    from tbempy import ThreeD
    rng = np.random.default_rng(n_obs)
    locs, nrm, w = clustered(401, 7)
    ol = rng.uniform(-1, 1, (n_obs, 3))
    on = np.tile([0.0, 0.0, 1.0], (n_obs, 1))
    K = ThreeD.ElasticTraction(1.0, 0.25)
    x = rng.uniform(-1, 1, 3 * len(locs))
    y = ThreeD.DirectOperator(K, ol, on, locs, nrm, w).apply(x)
    ref = oracle.direct("ElasticTraction", ol, on, locs, nrm, w, x)
    assert np.linalg.norm(y - ref) < 1e-11 * np.linalg.norm(ref)
