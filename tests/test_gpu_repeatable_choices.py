"""Threads per target are chosen by timing at construction, and the choice sets
an order of summation: operators whose variants tie must not fall to another
one from construction to construction.

The plain form is deterministic but for these choices.  Its pseudo-inverses turn
another order at the check surfaces into 1e-9 to 1e-8 of the result; another
order in the near field stays FP64 rounding (1e-15).  So repeated constructions
agree to 1e-12.  The precision form reports its near field's choice."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CONSTRUCTIONS = 8


@pytest.mark.parametrize("dim,kernel,size,order,leaf", [
    (2, "LaplaceSingle", 12575, 16, 32), (2, "ElasticTraction", 6354, 24, 32), (3, "LaplaceSingle", 14, 75, 50),
    (3, "ElasticDisplacement", 23, 99, 40), (3, "LaplaceSingle", 20, 152, 50)])
def test_plain_operators_repeat(dim, kernel, size, order, leaf):
    from tbempy import ThreeD, TwoD, meshes
    mod = TwoD if dim == 2 else ThreeD
    if dim == 3:
        pts, nrm, w = meshes.fault_points(size)[:3]
    else:
        a = 2.0 * np.pi * (np.arange(size) + 0.5) / size
        r = 1.0 + 0.1 * np.cos(5 * a)
        pts = np.ascontiguousarray(np.stack([r * np.cos(a), r * np.sin(a)], axis=1))
        nrm = np.ascontiguousarray(np.stack([np.cos(a), np.sin(a)], axis=1))
        w = np.full(size, 2.0 * np.pi / size)
    K = getattr(mod, kernel)
    K = K(1.0, 0.25) if kernel.startswith("Elastic") else K()
    y = []
    for _ in range(CONSTRUCTIONS):
        op = ThreeD.FMMOperator(K, pts, nrm, pts, nrm, w, ThreeD.FMMConfig(0.3, order, leaf, 0.05, False))
        y.append(op.apply(np.random.default_rng(4).uniform(-1, 1, op.n_cols())))
    assert max(np.linalg.norm(v - y[0]) for v in y) <= 1e-12 * np.linalg.norm(y[0])


@pytest.mark.parametrize("kernel,size,leaf", [("ElasticDisplacement", 24, 30), ("ElasticTraction", 40, 64),
                                              ("LaplaceSingle", 40, 40)])
def test_near_field_choice_repeats(kernel, size, leaf):
    from tbempy import ThreeD, meshes
    pts, nrm, w = meshes.fault_points(size)[:3]
    K = getattr(ThreeD, kernel)
    K = K(1.0, 0.25) if kernel.startswith("Elastic") else K()
    picks = {ThreeD.FMMOperator(K, pts, nrm, pts, nrm, w, ThreeD.FMMConfig(0.3, 152, leaf, 0.05, False),
                                precision="mixed").p2p_block() for _ in range(CONSTRUCTIONS)}
    assert len(picks) == 1
