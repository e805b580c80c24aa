"""Many right-hand sides in blocks of 16 (the batched form's near field and
points-to-check-surface passes): counts that fill the blocks, leave one over and
leave a ragged block, for batches on both sides of the rule that keeps the sums
in registers or in shared memory, against the FP64 direct sum.

Tolerance: the expansions of order 152 at MAC 0.3 and FP32 products reach 3e-7
on spheres in both layers; 2e-6 of the norm.  A right-hand side alone takes the
other kernel: the two agree to FP32 rounding of at most 128-term partial sums,
1e-6 of the norm."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


def batch(levels):
    from tbempy import meshes
    rng = np.random.default_rng(2)
    L, N, W, off = [], [], [], [0]
    for lev in levels:
        l, n, w = meshes.sphere_points(lev)
        r, c = rng.lognormal(0.0, 0.5), rng.uniform(-100.0, 100.0, 3)
        L.append(l * r + c)
        N.append(n)
        W.append(w * r * r)
        off.append(off[-1] + len(l))
    return np.concatenate(L), np.concatenate(N), np.concatenate(W), np.asarray(off, dtype=np.int64)


@pytest.mark.parametrize("kernel,levels", [("LaplaceSingle", (2, 3, 2)), ("LaplaceDouble", (2, 3, 2)),
                                           ("LaplaceDouble", (3, 3, 2, 3, 3)), ("LaplaceSingle", (4, 3, 4, 4))])
@pytest.mark.parametrize("n_rhs", [16, 17, 33, 37])
def test_blocks_of_right_hand_sides(kernel, levels, n_rhs):
    from tbempy import ThreeD
    L, N, W, off = batch(levels)
    op = ThreeD.BatchedFMMOperator(getattr(ThreeD, kernel)(), L, N, W, off, ThreeD.FMMConfig(0.3, 152, 128, 0.05, False))
    x = np.random.default_rng(n_rhs).uniform(-1, 1, (n_rhs, len(L)))
    y = op.apply(x)
    for r in sorted({0, 15, 16, n_rhs - 1} & set(range(n_rhs))):
        alone = op.apply(x[r])
        assert np.linalg.norm(y[r] - alone) <= 1e-6 * np.linalg.norm(alone)
        if r in (0, n_rhs - 1):
            a, b = off[0], off[1]  # the first mesh
            ref = oracle.direct(kernel, L[a:b], N[a:b], L[a:b], N[a:b], W[a:b], x[r, a:b])
            assert np.linalg.norm(y[r, a:b] - ref) <= 2e-6 * np.linalg.norm(ref)
            a, b = off[-2], off[-1]
            ref = oracle.direct(kernel, L[a:b], N[a:b], L[a:b], N[a:b], W[a:b], x[r, a:b])
            assert np.linalg.norm(y[r, a:b] - ref) <= 2e-6 * np.linalg.norm(ref)
