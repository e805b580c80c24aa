"""The precision form's outputs keep their order of summation: forward and
transposed applies and the geometry gradients of operators on one and on two
surfaces, against values that were written down before the passes were last
rewritten (golden/precision_outputs.npz, from the tree at commit 9798733).

The threads per target are given, so that only the passes themselves are
compared, and the outputs are means of six calls: the passes' atomic FP32 sums
reorder from call to call, a changed order of summation stays.  Tolerance: four
times the largest difference of such means between six constructions of that
tree, stored beside every output."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "precision_outputs.npz")

CALLS = 6

# kernel, surface, its size, observers on a plane above it (0: the same points), order, points per leaf
OPERATORS = {
    "single_two_surfaces": ("LaplaceSingle", "warped_fault", 20, 1600, 296, 64),
    "displacement_two_surfaces": ("ElasticDisplacement", "warped_fault", 15, 1100, 296, 64),
    "single_sphere": ("LaplaceSingle", "sphere", 2, 0, 152, 30),
    "double_spiral": ("LaplaceDouble", "spiral", 20, 0, 152, 64),
    "double_spiral_small": ("LaplaceDouble", "spiral", 14, 0, 152, 64),
    "traction_fault": ("ElasticTraction", "fault", 14, 0, 296, 40),
}


def outputs(name):
    from tbempy import ThreeD, meshes
    kernel, surface, size, n_obs, order, leaf = OPERATORS[name]
    if surface == "sphere":
        src, nrm, w = meshes.sphere_points(size)
    elif surface == "spiral":  # 6 size^2 + 1 points spread over the unit sphere
        i = np.arange(6 * size * size + 1) + 0.5
        c, a = 1.0 - 2.0 * i / len(i), np.pi * (1.0 + 5.0 ** 0.5) * i
        r = np.sqrt(1.0 - c * c)
        src = np.ascontiguousarray(np.stack([r * np.cos(a), r * np.sin(a), c], axis=1))
        nrm, w = src.copy(), np.full(len(i), 4.0 * np.pi / len(i))
    else:
        v, t, _ = meshes.dipping_fault(size, 45.0)
        if surface == "warped_fault":
            v = v.copy()
            v[:, 2] += 0.05 * np.sin(3 * v[:, 0]) * np.cos(2 * v[:, 1])
        src, nrm, w = meshes.points_from_mesh(v, t)
    rng = np.random.default_rng(8)
    obs, onrm = src, nrm
    if n_obs:
        obs = np.ascontiguousarray(np.concatenate([rng.uniform(-3, 3, (n_obs, 2)), np.zeros((n_obs, 1))], axis=1))
        onrm = np.tile([0.0, 0.0, 1.0], (n_obs, 1))
    K = getattr(ThreeD, kernel)
    op = ThreeD.FMMOperator(K(1.0, 0.25) if kernel.startswith("Elastic") else K(), obs, onrm, src, nrm, w,
                            ThreeD.FMMConfig(0.3, order, leaf, 0.05, False), precision="mixed", p2p_block=4, p2m_block=4)
    assert op.m2l_ranks()[0] > 0
    x, z = rng.uniform(-1, 1, op.n_cols()), rng.uniform(-1, 1, op.n_rows())
    mean = {}
    for _ in range(CALLS):
        out = {"y": op.apply(x), "transposed": op.apply_adjoint(z)}
        out.update(op.source_gradients(x, z))
        out.update(op.observation_gradients(x, z))
        for k, v in out.items():
            mean[k] = mean.get(k, 0.0) + np.asarray(v) / CALLS
    return {k: v for k, v in mean.items() if np.any(v)}


@pytest.mark.parametrize("name", sorted(OPERATORS))
def test_outputs_are_those_written_down(name):
    with np.load(GOLDEN) as g:
        gold = {k: g[k] for k in g.files if k.startswith(name + "/")}
    out = outputs(name)
    assert {k.split("/")[1] for k in gold} == set(out)
    off = {}
    for k, v in out.items():
        ref = gold["%s/%s" % (name, k)]
        off[k] = np.linalg.norm(v - ref) / np.linalg.norm(ref) / float(gold["%s/%s/spread" % (name, k)])
    assert max(off.values()) <= 4.0, off
