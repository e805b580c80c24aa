"""The gradient passes where source lists are long: a dense cluster among
scattered points, whose leaves see thousands of sources (a whole CTA per target)
beside lists of a few dozen (a warp per target), against the direct gradient
pass.

Tolerance: FP64 compressed expansions of order 152 reach 1e-6 in the value and
lose one to two digits in a derivative: 1e-4 of the norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3001, 6002])
def test_long_lists_match_the_direct_pass(n):
    from tbempy import ThreeD
    rng = np.random.default_rng(5)
    a = rng.uniform(-1, 1, (n // 20, 3))
    b = 0.02 * rng.normal(size=(n - len(a), 3)) + [0.3, 0.2, -0.1]
    locs = np.concatenate([a, b])
    nrm = rng.normal(size=locs.shape)
    nrm /= np.linalg.norm(nrm, axis=1)[:, None]
    w = rng.uniform(0.5, 1.0, n)
    K = ThreeD.LaplaceSingle()
    op = ThreeD.FMMOperator(K, locs, nrm, locs, nrm, w, ThreeD.FMMConfig(0.3, 152, 60, 0.05, False),
                            precision="fp64_compressed")
    x, r = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    d = ThreeD.direct_gradients(K, locs, nrm, locs, nrm, w, x, r)
    for key, v in dict(op.source_gradients(x, r), **op.observation_gradients(x, r)).items():
        if np.abs(d[key]).max() > 0:
            assert np.linalg.norm(v - d[key]) <= 1e-4 * np.linalg.norm(d[key])
        else:
            assert np.abs(v).max() == 0
