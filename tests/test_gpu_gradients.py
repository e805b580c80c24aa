"""The kernels' written-out derivatives (the direct gradient pass and the FMM's
gradient passes share them) against central differences of L = r^T A x, for
every 3D kernel, in every position and normal, and the FMM passes against the
direct pass at point counts that leave the pass's eight-target CTAs and its
sixteen threads per target with remainders.

Tolerances: the point sets are at least 1 apart, so with h = 1e-5 the
differences' truncation (h^2 times third derivatives of order 10) and rounding
(1e-16 |L| / h) are below 1e-8 of the largest derivative: 1e-6 is asserted.
The FP64 compressed form follows the direct pass to its expansions' accuracy
(about 1e-7 in the value, one to two digits less in a derivative): 1e-4.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KERNELS = ["LaplaceSingle", "LaplaceDouble", "ElasticDisplacement", "ElasticTraction",
           "ElasticAdjointTraction", "ElasticHypersingular", "IdentityScalar"]


def kernel(name):
    from tbempy import ThreeD
    k = getattr(ThreeD, name)
    return k(1.3, 0.2) if name.startswith("Elastic") else k()


def cloud(rng, n, shift):
    nrm = rng.normal(size=(n, 3))
    return rng.uniform(0, 1, (n, 3)) + [shift, 0, 0], nrm / np.linalg.norm(nrm, axis=1)[:, None]


@pytest.mark.parametrize("name", KERNELS)
def test_direct_gradients_match_central_differences(name):
    from tbempy import ThreeD
    K = kernel(name)
    rng = np.random.default_rng(3)
    ol, on = cloud(rng, 5, 2.0)
    sl, sn = cloud(rng, 4, 0.0)
    w = rng.uniform(0.5, 1.0, len(sl))
    x = rng.uniform(-1, 1, K.tensor_dim * len(sl))
    r = rng.uniform(-1, 1, K.tensor_dim * len(ol))
    args = {"obs_locs": ol, "obs_normals": on, "src_locs": sl, "src_normals": sn}

    def loss(**kw):
        a = dict(args, **kw)
        return float(r @ ThreeD.DirectOperator(K, a["obs_locs"], a["obs_normals"], a["src_locs"],
                                               a["src_normals"], w).apply(x))

    g = ThreeD.direct_gradients(K, ol, on, sl, sn, w, x, r)
    h = 1e-5
    num = {}
    for key, v in args.items():
        num[key] = np.zeros_like(v)
        for i in np.ndindex(*v.shape):
            d = np.zeros_like(v)
            d[i] = h
            num[key][i] = (loss(**{key: v + d}) - loss(**{key: v - d})) / (2 * h)
    for a, b in (("obs_locs", "src_locs"), ("obs_normals", "src_normals")):
        scale = max(np.abs(num[a]).max(), np.abs(num[b]).max(), 1e-300)
        if name == "IdentityScalar" or (a == "obs_normals" and scale < 1e-9):
            scale = 1.0
        for key in (a, b):
            assert np.abs(g[key] - num[key]).max() <= 1e-6 * scale


@pytest.mark.parametrize("name", ["LaplaceDouble", "ElasticTraction", "ElasticHypersingular"])
@pytest.mark.parametrize("n_obs,n_src,leaf", [(517, 389, 23), (803, 641, 37)])
def test_fmm_gradients_match_the_direct_pass_at_ragged_sizes(name, n_obs, n_src, leaf):
    from tbempy import ThreeD
    K = kernel(name)
    rng = np.random.default_rng(4)
    (ol, on), (sl, sn) = cloud(rng, n_obs, 0.3), cloud(rng, n_src, 0.0)
    w = rng.uniform(0.5, 1.0, n_src)
    op = ThreeD.FMMOperator(K, ol, on, sl, sn, w, ThreeD.FMMConfig(0.3, 296, leaf, 0.05, False),
                            precision="fp64_compressed")
    x = rng.uniform(-1, 1, op.n_cols())
    r = rng.uniform(-1, 1, op.n_rows())
    d = ThreeD.direct_gradients(K, ol, on, sl, sn, w, x, r)
    g = dict(op.source_gradients(x, r), **op.observation_gradients(x, r))
    for key, v in g.items():
        if np.abs(d[key]).max() > 0:
            assert np.linalg.norm(v - d[key]) <= 1e-4 * np.linalg.norm(d[key])
        else:
            assert np.abs(v).max() == 0
