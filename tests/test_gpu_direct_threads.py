"""The direct sum's threads per target (8, 16 or 32 by the number of points, one
number for all CTAs): point counts that take each of them on 152 SMs, with
remainders, for one and three right-hand sides, and the entry that allocates
nothing up to a point count whose work items fit its scratch with fewer threads
only.

Tolerance: two FP64 sums of n terms of either sign differ by less than n 2^-53
of the sum of magnitudes: 1e-11 of the norm for the few hundred sources here."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


def cloud(n, seed):
    rng = np.random.default_rng(seed)
    nrm = rng.normal(size=(n, 3))
    return rng.uniform(-1, 1, (n, 3)), nrm / np.linalg.norm(nrm, axis=1)[:, None], rng.uniform(0.5, 1.0, n)


@pytest.mark.parametrize("kernel", ["LaplaceDouble", "ElasticTraction"])
@pytest.mark.parametrize("n_obs", [7, 601, 1177, 2401, 4705, 4901, 12001])
@pytest.mark.parametrize("n_rhs", [1, 3])
def test_direct_sum(kernel, n_obs, n_rhs):
    from tbempy import ThreeD
    ol, on, _ = cloud(n_obs, 1)
    sl, sn, w = cloud(259, 2)
    K = getattr(ThreeD, kernel)
    K = K(1.0, 0.25) if kernel.startswith("Elastic") else K()
    op = ThreeD.DirectOperator(K, ol, on, sl, sn, w)
    x = np.random.default_rng(3).uniform(-1, 1, (n_rhs, op.n_cols()))
    y = op.apply(x)
    for r in range(n_rhs):
        ref = oracle.direct(kernel, ol, on, sl, sn, w, x[r])
        assert np.linalg.norm(y[r] - ref) <= 1e-11 * np.linalg.norm(ref)


@pytest.mark.parametrize("n_obs", [2401, 4901, 1_000_003, 3_000_001])
def test_allocation_free_entry_with_many_observers(n_obs):
    torch = pytest.importorskip("torch")
    from tbempy import _lib
    g = torch.Generator(device="cuda").manual_seed(5)
    new = lambda *s: torch.rand(s, generator=g, device="cuda", dtype=torch.float64)
    ol, on, sl, sn, w, x = new(n_obs, 3), new(n_obs, 3), new(11, 3) + 2.0, new(11, 3), new(11), new(11)
    y = [torch.full((n_obs,), float("nan"), device="cuda", dtype=torch.float64) for _ in range(2)]
    p = lambda t: C.c_void_p(t.data_ptr())
    for name, out in zip(("tbem_direct_apply_noalloc", "tbem_direct_apply"), y):
        _lib.check(getattr(_lib.lib(), name)(0, None, p(ol), p(on), n_obs, p(sl), p(sn), p(w), 11, p(x), p(out), 1, None))
    torch.cuda.synchronize()
    assert float((y[0] - y[1]).abs().max()) <= 1e-11 * float(y[1].abs().max())
