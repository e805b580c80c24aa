"""The CSR apply where lanes per row follow the longest row (a few rows of
hundreds to hundreds of thousands of entries among short ones) and where long
mean rows take more lanes in launches of one or four right-hand sides only; the
counts of right-hand sides mix such launches with others.

Tolerance: sums of n products in any order differ by at most 2 n eps sum |a x|
(eps 2^-53 each for product and sum)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_rows,short,long,every", [
    (50000, 12, 5000, 1000), (100003, 50, 500, 100), (60000, 20, 100000, 60000), (40009, 300, 300, 1),
    (2011, 900, 900, 1), (17, 3, 4000, 17)])
@pytest.mark.parametrize("n_rhs", [1, 4, 5, 7])
def test_csr_apply_with_long_rows(n_rows, short, long, every, n_rhs):
    from tbempy import ThreeD
    rng = np.random.default_rng(n_rows)
    count = np.full(n_rows, short)
    count[every - 1::every] = long
    rows = np.concatenate([[0], np.cumsum(count)]).astype(np.int64)
    n_cols = 1201
    cols = rng.integers(0, n_cols, rows[-1])
    vals = rng.normal(size=rows[-1])
    op = ThreeD.SparseOperator(n_rows, n_cols, vals, cols, rows)
    x = rng.normal(size=(n_rhs, n_cols))
    y = op.apply(x if n_rhs > 1 else x[0]).reshape(n_rhs, n_rows)
    for r in range(n_rhs):
        prod = vals * x[r, cols]
        ref = np.add.reduceat(prod, rows[:-1])
        mag = np.add.reduceat(np.abs(prod), rows[:-1])
        # the reference's own sums are rounded as well
        assert np.all(np.abs(y[r] - ref) <= 4 * count * 2.0 ** -53 * mag)
