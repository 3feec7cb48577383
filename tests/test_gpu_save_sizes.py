"""Save steps of fields on either side of 2^16 points, where the mu/M kernel of a
save step changes its points per block, against the oracle."""
import numpy as np
import pytest

from test_gpu_save import RTOL, _close, _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
@pytest.mark.parametrize("dim,shape", [(1, (65535,)), (1, (65536,)), (2, (31, 33)), (2, (257, 256)), (3, (9, 33, 31)),
                                       (3, (41, 40, 42))])
def test_save_step_on_either_side(dim, shape, precision):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from oracle.oracle import OracleStepper
    from phasefield5d_b200.stepper import Stepper
    prob = _problem(dim, shape)
    st, ost = Stepper.from_problem(prob, precision=precision), OracleStepper.from_problem(prob)
    # the tolerances of test_gpu_save for each form
    rt, rv, rf = (RTOL, 1e-8, 1e-12) if precision == "fp64" else (1e-5, 1e-2, 1e-5)
    g, r = st.step_save(), ost.step_save()
    for key in ("mass", "comp_min", "comp_max", "max_change"):
        assert _close(g[key], r[key], np.abs(r[key]), rt), (key, g[key], r[key])
    assert _close(g["comp_var"], r["comp_var"], np.abs(r["comp_var"]), rv)
    # formed from the save step's own mu and M: rounding noise of sums that cancel
    assert _close(g["total_flux"], r["total_flux"], r["flux_abs"], rf), (g["total_flux"], r["flux_abs"])
    assert _close(g["net"], r["net"], np.prod(shape) * r["xdotmax"], rf)
    st.close()
