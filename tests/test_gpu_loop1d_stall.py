"""A launch of the 1D step loop whose blocks give up their waits for one another:
it ends with PF5D_FLAG_STALLED, the field and the state are those before the
launch as a whole (blocks that got their messages must not store while others
did not), callers get an error instead of a halt, and a reset starts over."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _raw(st):
    from phasefield5d_b200 import _lib
    s = _lib.StepState()
    _lib.check(st.L.pf5d_stepper_state(st.h, ctypes.byref(s), st._s()))
    return s


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
@pytest.mark.parametrize("n", [203, 1280, 4112])
def test_stalled_launch_changes_nothing(n, precision):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from phasefield5d_b200 import _lib, workload as W
    from phasefield5d_b200.stepper import Stepper
    cfg = W.SolveConfig(system_dim=1, initial_composition=(0.1, 0.2, 0.2, 0.25), resolution=0.05,
                        kappa_value=5e-16, mw=4, ppw=16, shape=(n,), n_k=500, fluctuation=2e-2)
    prob = W.build_problem(cfg)
    st, ref = (Stepper.from_problem(prob, precision=precision) for _ in range(2))
    st.advance(4)
    ref.advance(4)
    before, field = _raw(st), st.field()
    assert before.flags == 0 and torch.equal(field, ref.field())
    stalls = 0
    for steps in (1, 2, 3, 5, 8, 40):
        st.set_wait_limit(0.0)               # one look at each message
        st.advance(steps)
        s = _raw(st)
        st.set_wait_limit(2.0)
        if s.flags & _lib.FLAG_STALLED:
            stalls += 1
            assert s.halted and torch.equal(st.field(), field)
            assert (s.dt, s.time, s.xdotmax, s.step) == (before.dt, before.time, before.xdotmax,
                                                         before.step)
            with pytest.raises(RuntimeError, match="stalled"):
                st.run(1)                    # halted: no step
            with pytest.raises(RuntimeError, match="stalled"):
                st.state()
        # from the start again, as far as the reference solve
        st.X.copy_(torch.from_numpy(np.ascontiguousarray(prob.X_init)))
        st.reset(prob.dt0)
        st.advance(4)
        assert torch.equal(st.field(), field) and _raw(st).flags == 0
    assert stalls >= 1
    st.close()
    ref.close()


def test_wait_limit_range():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from phasefield5d_b200 import workload as W
    from phasefield5d_b200.stepper import Stepper
    st = Stepper.from_problem(W.build_problem(W.SolveConfig(
        system_dim=1, initial_composition=(0.1, 0.2, 0.2, 0.25), resolution=0.05, kappa_value=5e-16,
        mw=4, ppw=16, shape=(40,), n_k=500)))
    for bad in (-1.0, float("nan"), 1e9):
        with pytest.raises(ValueError):
            st.set_wait_limit(bad)
    st.close()
