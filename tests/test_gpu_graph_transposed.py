"""A captured forward graph of a precision-form operator replays after
transposed applies and gradient passes of the same operator: those keep every
buffer that the graph's kernels address.

The operator has observers on a plane over a warped fault, where the output
ranks round up to more than the input ranks (the case in which buffers sized
for one direction would not do for the other).  Tolerance: replays repeat up to
the order of atomic FP32 sums, 1e-6 of the norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_rhs", [1, 3])
def test_graph_after_transposed_applies(n_rhs):
    torch = pytest.importorskip("torch")
    from tbempy import ThreeD, meshes
    v, t, _ = meshes.dipping_fault(17, 45.0)
    v = v.copy()
    v[:, 2] += 0.05 * np.sin(3 * v[:, 0]) * np.cos(2 * v[:, 1])
    src, nrm, w = meshes.points_from_mesh(v, t)
    rng = np.random.default_rng(5)
    obs = np.ascontiguousarray(np.concatenate([rng.uniform(-3, 3, (1300, 2)), np.zeros((1300, 1))], axis=1))
    op = ThreeD.FMMOperator(ThreeD.ElasticDisplacement(1.0, 0.25), obs, np.tile([0.0, 0.0, 1.0], (1300, 1)), src, nrm, w,
                            ThreeD.FMMConfig(0.3, 296, 64, 0.05, False), precision="mixed")
    ri, ro = op.m2l_ranks()
    assert (ro + 63) // 64 > (ri + 63) // 64
    x = torch.tensor(rng.uniform(-1, 1, (n_rhs, op.n_cols())), device="cuda")
    y = torch.zeros((n_rhs, op.n_rows()), dtype=torch.float64, device="cuda")
    z = torch.tensor(rng.uniform(-1, 1, (n_rhs, op.n_rows())), device="cuda")
    torch.cuda.synchronize()
    g = ThreeD.FMMGraph([op], [x], [y], n_rhs=n_rhs)
    torch.cuda.synchronize()
    ref = y.clone()
    others = []
    for _ in range(2):
        op.apply_adjoint(z)
        if n_rhs == 1:
            op.source_gradients(x[0], z[0])
        others.append(torch.full((1 << 20,), 3.0, device="cuda"))  # would take freed memory
        x.uniform_(-1, 1)
        y.zero_()
        torch.cuda.synchronize()
        g.launch()
        torch.cuda.synchronize()
        ref = op.apply(x)
        assert float((y - ref).norm() / ref.norm()) < 1e-6
        assert all(bool((o == 3.0).all()) for o in others)


@pytest.mark.parametrize("precision", ["fp64", "mixed", "fp64_compressed"])
def test_graph_after_applies_of_more_right_hand_sides(precision):
    """Applies that outgrow the work buffers keep those that a live graph
    addresses; without a live graph they are freed."""
    torch = pytest.importorskip("torch")
    from tbempy import ThreeD, meshes
    locs, nrm, w = meshes.sphere_points(3)
    op = ThreeD.FMMOperator(ThreeD.LaplaceSingle(), locs, nrm, locs, nrm, w,
                            ThreeD.FMMConfig(0.3, 152, 50, 0.05, False), precision=precision)
    n = len(locs)
    x = torch.rand(n, dtype=torch.float64, device="cuda")
    y = torch.zeros(n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    g = ThreeD.FMMGraph([op], [x], [y])
    many = torch.rand((9, n), dtype=torch.float64, device="cuda")
    tol = {"fp64": 0.0, "mixed": 1e-6, "fp64_compressed": 1e-13}[precision]  # the atomic sums' order

    def replays():
        x.uniform_(-1, 1)
        y.zero_()
        torch.cuda.synchronize()
        g.launch()
        torch.cuda.synchronize()
        ref = op.apply(x)
        torch.cuda.synchronize()
        return float((y - ref).norm()) <= tol * float(ref.norm())

    assert replays()
    for n_rhs in (3, 9):
        op.apply(many[:n_rhs])
        op.apply_adjoint(many[:n_rhs])
        torch.cuda.synchronize()
        filler = torch.full((1 << 22,), 3.0, device="cuda")  # would take freed memory
        assert replays() and bool((filler == 3.0).all())
    del g
    before = torch.cuda.mem_get_info()[0]
    ref = op.apply(x)  # frees what the graph had kept
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] >= before
    assert torch.isfinite(ref).all()
