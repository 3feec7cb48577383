"""Reading the field of a solve that runs on a stream of its own: what the
caller's stream does with the tensor comes after the steps enqueued so far, and
the tensor's memory is not written while that stream still uses it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _problem(shape):
    from phasefield5d_b200 import workload as W
    cfg = W.batched_configs(1, seed=5, steps=40)[0]
    cfg.shape, cfg.system_dim = shape, len(shape)
    return W.build_batched_problems([cfg])[0][0]


@pytest.mark.parametrize("form", ["fp64", "fp32c", "batch"])
def test_field_waits_for_the_steps(torch_cuda, form):
    torch = torch_cuda
    from phasefield5d_b200.batch import BatchStepper
    from phasefield5d_b200.stepper import Stepper
    prob, steps = _problem((256, 256)), 3000            # some 50 ms of queued steps
    own = torch.cuda.Stream()
    with torch.cuda.stream(own):
        if form == "batch":
            st = BatchStepper([prob], stream=own, autotune=False)
        else:
            st = Stepper.from_problem(prob, precision=form, stream=own, autotune=False)
    read = (lambda: st.field(0)) if form == "batch" else st.field
    st.advance(steps)
    got = read().cpu().numpy()                          # on the default stream
    torch.cuda.synchronize()
    with torch.cuda.stream(own):
        want = read().cpu().numpy()
    assert np.array_equal(got, want)
    if form == "fp64":
        st.advance(steps)
        got = st.rate().clone()
        torch.cuda.synchronize()
        assert torch.equal(got, st.rate())
    # memory freed on the default stream, still read there, is not overwritten
    torch.cuda.synchronize()
    del got
    a = torch.full((*prob.shape, 4), 7.0, dtype=torch.float64, device="cuda")
    other = torch.empty_like(a)
    torch.cuda._sleep(50_000_000)
    other.copy_(a)
    del a
    out = read()
    torch.cuda.synchronize()
    assert bool((other == 7.0).all()) and torch.isfinite(out).all()
    st.close()
