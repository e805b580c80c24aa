"""The CSR apply where its row walk can go wrong: empty rows, rows of one entry
below, at and above a step of every lane count, one very long row, row counts
that leave a warp's last set ragged, and enough rows for the narrow lanes; one
and several right-hand sides.

Tolerance: a sum of n products in any order differs from another by at most
2 n eps sum |a x| (n the row's entries, eps 2^-53 each for product and sum)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_rows,lengths", [
    (1, [0]), (1, [7]), (3, [0, 1, 5000]), (33, [3]), (37, [0, 1, 15, 16, 17, 31, 32, 33]),
    (1000, [63, 64, 65, 0, 127, 128, 129]), (5000, [12, 0, 30]), (170001, [50, 20, 0, 71]), (90007, [9, 40])])
@pytest.mark.parametrize("n_rhs", [1, 3])
def test_csr_apply_at_step_edges(n_rows, lengths, n_rhs):
    from tbempy import ThreeD
    rng = np.random.default_rng(n_rows)
    count = rng.choice(lengths, n_rows)
    count[:len(lengths)] = lengths[:n_rows]
    rows = np.concatenate([[0], np.cumsum(count)]).astype(np.int64)
    n_cols = 977
    cols = rng.integers(0, n_cols, rows[-1])
    vals = rng.normal(size=rows[-1])
    op = ThreeD.SparseOperator(n_rows, n_cols, vals, cols, rows)
    x = rng.normal(size=(n_rhs, n_cols))
    y = op.apply(x if n_rhs > 1 else x[0]).reshape(n_rhs, n_rows)
    for r in range(n_rhs):
        prod = vals * x[r, cols]
        total = np.concatenate([[0.0], np.cumsum(prod.astype(np.longdouble))])
        mag = np.concatenate([[0.0], np.cumsum(np.abs(prod))])
        ref = (total[rows[1:]] - total[rows[:-1]]).astype(np.float64)
        # the reference's own running sums round at the size of the whole array
        eps = float(np.finfo(np.longdouble).eps)
        bound = 2 * count * 2.0 ** -53 * (mag[rows[1:]] - mag[rows[:-1]]) * (1 + 1e-9) + 2 * eps * mag[-1] * len(prod) ** 0.5
        assert np.all(np.abs(y[r] - ref) <= bound + 1e-300)
    assert np.array_equal(op._cols, cols)
