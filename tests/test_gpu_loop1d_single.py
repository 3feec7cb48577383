"""A single step of a 1D solve around the length from which its kernels run apart
(10240 points): the same bits as in the loop, and no slower than the stages."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _stepper(n, precision):
    from phasefield5d_b200 import workload as W
    from phasefield5d_b200.stepper import Stepper
    return Stepper.from_problem(W.build_problem(W.SolveConfig(
        system_dim=1, initial_composition=(0.1, 0.2, 0.2, 0.25), resolution=0.05, kappa_value=5e-16,
        mw=4, ppw=16, shape=(n,), n_k=500, fluctuation=2e-2)), precision=precision)


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
@pytest.mark.parametrize("n", [10240, 10241, 16384])
def test_single_steps_equal_one_launch(torch_cuda, n, precision):
    a, b = _stepper(n, precision), _stepper(n, precision)
    for _ in range(6):
        a.advance(1)
    b.advance(6)
    assert a.state() == b.state() and a.state()["step"] == 6
    assert torch_cuda.equal(a.field(), b.field())
    a.close()
    b.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
def test_single_step_of_a_long_solve(torch_cuda, precision):
    """At most 1.1 times its four kernels, launched stage by stage (the loop: 1.16
    and 1.28 times)."""
    from phasefield5d_b200 import _lib
    st = _stepper(16384, precision)

    def stages():
        for stage in (_lib.STAGE_FFT_FWD, _lib.STAGE_RATE, _lib.STAGE_UPDATE):
            st.launch_stage(stage)

    def us(call):
        out = []
        for _ in range(30):
            a, b = (torch_cuda.cuda.Event(enable_timing=True) for _ in range(2))
            torch_cuda.cuda._sleep(400_000)
            a.record()
            call()
            b.record()
            torch_cuda.cuda.synchronize()
            out.append(a.elapsed_time(b) * 1e3)
        return float(np.median(out))

    st.advance(1)
    apart = us(stages)
    assert us(lambda: st.advance(1)) <= 1.1 * apart
    st.close()
