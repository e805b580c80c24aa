"""The FP64 compressed form's digit planes are a choice: on a GPU that other
work has filled, the operator leaves them out and keeps the FP64 pipe, with the
same results and without a failure.

An allocation stands for the other work: it leaves 6 GB, and the planes of the
operator here take 0.7 GB, more than a sixteenth."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_planes_are_left_out_on_a_filled_gpu():
    torch = pytest.importorskip("torch")
    from tbempy import ThreeD, meshes
    locs, nrm, w = meshes.sphere_points(3)

    def operator(path):
        return ThreeD.FMMOperator(ThreeD.LaplaceSingle(), locs, nrm, locs, nrm, w,
                                  ThreeD.FMMConfig(0.3, 152, 30, 0.05, False), precision="fp64_compressed", m2l_path=path)

    x = np.random.default_rng(3).uniform(-1, 1, len(locs))
    pipe = operator(4)
    y = pipe.apply(x)
    roomy = operator(0)
    roomy.apply(x)
    assert roomy.last_launches() == pipe.last_launches() + 1  # the launch that splits the coefficients
    planes = torch.cuda.mem_get_info()[0]
    del roomy
    planes = torch.cuda.mem_get_info()[0] - planes  # the operator with its planes
    ThreeD.clear_setup_cache()
    filler = torch.empty(torch.cuda.mem_get_info()[0] - (6 << 30), dtype=torch.uint8, device="cuda")
    try:
        free = torch.cuda.mem_get_info()[0]
        tight = operator(0)
        taken = free - torch.cuda.mem_get_info()[0]
        y_tight = tight.apply(x)
        launches = tight.last_launches()
    finally:
        del filler
        torch.cuda.empty_cache()
    assert launches == pipe.last_launches()
    assert taken < planes - (1 << 29)
    assert np.linalg.norm(y_tight - y) <= 1e-13 * np.linalg.norm(y)  # the order of the atomic sums
