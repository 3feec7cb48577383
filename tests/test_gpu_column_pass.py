"""The column pass of the elastic term for every transform length, with whole
lines of columns per block (3D spectra) and with two (2D), column counts that do
not divide, against the oracle's scipy transforms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELD_RTOL = 1e-12      # the plain FP64 form's tolerance on X


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("n0", [8, 16, 32, 64, 128, 256, 512, 1024])
@pytest.mark.parametrize("rest", [(49, 101), (3, 5), (7,)])
def test_column_pass_matches_oracle(torch_cuda, n0, rest):
    from oracle.oracle import OracleStepper
    from phasefield5d_b200 import workload as W
    from phasefield5d_b200.stepper import Stepper
    shape = (n0, *rest)
    cfg = W.SolveConfig(system_dim=len(shape), initial_composition=(0.1, 0.2, 0.2, 0.25),
                        resolution=0.05, kappa_value=5e-16, mw=4, ppw=16, shape=shape, n_k=500,
                        fluctuation=2e-2)
    prob = W.build_problem(cfg)
    ref = OracleStepper.from_problem(prob)
    ref.step()
    st = Stepper.from_problem(prob, autotune=False)
    st.run(1)
    X = st.X.cpu().numpy()
    st.close()
    assert np.max(np.abs(X - ref.X)) <= FIELD_RTOL * np.max(np.abs(ref.X))
    moved = np.max(np.abs(ref.X - prob.X_init))
    assert np.max(np.abs(X - ref.X)) <= 1e-8 * moved      # the step itself, not only the field

    x32 = Stepper.from_problem(prob, autotune=False, precision="fp32c")
    x32.run(1)
    Y = x32.field().cpu().numpy()
    x32.close()
    assert np.max(np.abs(Y - ref.X)) <= 1e-4 * moved      # FP32 rates, FP32 transforms
