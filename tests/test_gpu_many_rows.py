"""Save steps of 3D fields with more rows along axis 1 than a grid's y dimension
has tiles of four."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
def test_save_step_with_a_long_middle_axis(precision):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from phasefield5d_b200 import workload as W
    from phasefield5d_b200.stepper import Stepper
    cfg = W.SolveConfig(system_dim=3, initial_composition=(0.1, 0.2, 0.2, 0.25), resolution=0.05,
                        kappa_value=5e-16, mw=4, ppw=16, shape=(2, 4 * 65535 + 9, 2), n_k=500,
                        include_cubic_anisotropy=False, fluctuation=2e-2)
    prob = W.build_problem(cfg)
    a, b = (Stepper.from_problem(prob, precision=precision) for _ in range(2))
    a.advance(2)
    for _ in range(2):
        d = b.step_save()
        assert not d["halted"]
    assert a.state() == b.state() and torch.equal(a.field(), b.field())
    # the total flux is a sum over faces that cancels, of the save step's own mu and M
    x, dx = prob.X_init, d["max_change"]
    assert np.all(np.abs(d["total_flux"]) <= 1e-5 * np.prod(x.shape[:-1]) * dx * prob.dx)
    a.close()
    b.close()
