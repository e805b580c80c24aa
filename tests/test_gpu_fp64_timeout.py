"""The bounded waits of the FP64 compressed form's tensor-core M2L, made to run
out on purpose (a budget of one cycle): the apply reports TBEM_ERR_TIMEOUT,
keeps reporting it, and leaves the device usable.  Nothing faults: the waits
end by themselves and return a status."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TIMEOUT = -5


def operator(path=0):
    from tbempy import ThreeD, meshes
    locs, nrm, w = meshes.sphere_points(3)
    return ThreeD.FMMOperator(ThreeD.LaplaceSingle(), locs, nrm, locs, nrm, w,
                              ThreeD.FMMConfig(0.3, 152, 50, 0.05, False), precision="fp64_compressed", m2l_path=path)


def test_wait_budget_exhausted_reports_timeout_and_device_stays_usable():
    torch = pytest.importorskip("torch")
    from tbempy._lib import TbemError
    op = operator()
    x = np.random.default_rng(0).uniform(-1, 1, op.n_cols())
    y_ok = op.apply(x)
    pipe = operator(4)  # the M2L on the FP64 pipe: no launch that splits the coefficients
    y_pipe = pipe.apply(x)
    assert op.last_launches() == pipe.last_launches() + 1
    op.set_wait_cycles(1)
    with pytest.raises(TbemError) as e:
        op.apply(x)
    assert e.value.code == TIMEOUT
    op.set_wait_cycles(0)
    for call in (lambda: op.apply(x), op.sync):  # the failure is latched
        with pytest.raises(TbemError) as e:
            call()
        assert e.value.code == TIMEOUT

    op2 = operator()  # device output: the apply returns, sync() reports
    op2.set_wait_cycles(1)
    op2.apply(torch.tensor(x, device="cuda"))
    with pytest.raises(TbemError) as e:
        op2.sync()
    assert e.value.code == TIMEOUT

    op3 = operator()  # the device is still usable
    y3 = op3.apply(x)
    op3.sync()
    # the split is error free to 2^-60 of the largest products: FP64 rounding apart
    assert np.linalg.norm(y3 - y_ok) <= 1e-13 * np.linalg.norm(y_ok)
    assert np.linalg.norm(y3 - y_pipe) <= 1e-13 * np.linalg.norm(y_pipe)
