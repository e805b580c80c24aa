"""An apply reads and writes this device's aligned buffers in place; buffers
that overlap, are not aligned to a double, or live on the host go through the
staging buffers.  All give the apply's result on separate buffers: bit for bit
in the plain form (1e-6 where the precision form's atomic sums reorder), in
chunks of right-hand sides too."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n_rhs", [1, 3])
@pytest.mark.parametrize("adjoint", [False, True])
def test_buffers_in_place_overlapping_unaligned_and_host(precision, n_rhs, adjoint):
    import torch
    from tbempy import ThreeD, _lib, meshes
    locs, nrm, w = meshes.sphere_points(2)
    n = len(locs)
    op = ThreeD.FMMOperator(ThreeD.LaplaceSingle(), locs, nrm, locs, nrm, w, ThreeD.FMMConfig(0.3, 152, 30, 0.05, False),
                            precision=precision)
    fn = _lib.lib().tbem_fmm_apply_adjoint if adjoint else _lib.lib().tbem_fmm_apply
    x = torch.from_numpy(np.random.default_rng(1).uniform(-1, 1, (n_rhs, n))).cuda()
    ref = (op.apply_adjoint(x) if adjoint else op.apply(x)).clone()
    tol = 0.0 if precision == "fp64" else 1e-6

    def close(y):
        torch.cuda.synchronize()
        return float((y.reshape(n_rhs, n) - ref).norm() / ref.norm()) <= tol

    def call(px, py):
        _lib.check(fn(op._h, C.c_void_p(px), C.c_void_p(py), n_rhs, C.c_void_p(1)))

    size = n_rhs * n
    buf = x.reshape(-1).clone()
    call(buf.data_ptr(), buf.data_ptr())  # the same buffer
    assert close(buf)
    buf = torch.zeros(size + 8, dtype=torch.float64, device="cuda")
    buf[:size] = x.reshape(-1)
    call(buf.data_ptr(), buf.data_ptr() + 8 * 8)  # overlapping
    assert close(buf[8:])
    raw = torch.zeros(8 * size + 16, dtype=torch.uint8, device="cuda")
    out = torch.zeros(8 * size + 16, dtype=torch.uint8, device="cuda")
    raw[4:4 + 8 * size] = x.reshape(-1).view(torch.uint8)
    call(raw.data_ptr() + 4, out.data_ptr() + 4)  # not aligned to a double
    torch.cuda.synchronize()
    assert close(out[4:4 + 8 * size].clone().view(torch.float64))
    hx, hy = x.cpu().numpy().copy(), np.zeros((n_rhs, n))
    call(hx.ctypes.data, hy.ctypes.data)
    assert close(torch.from_numpy(hy).cuda())
    dy = torch.zeros_like(x)
    call(hx.ctypes.data, dy.data_ptr())  # host input, device output
    assert close(dy)
