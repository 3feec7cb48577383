"""A step loop ends between its kernels, never inside one: the update that finds
the field out of bounds still writes every point, and a rate evaluation that
meets non-finite compositions runs in every block and leaves field, dt, time and
step as they were.  Sizes give several rounds of blocks (batch: 4096 update
chunks on 148 SMs) and blocks with and without a bad point."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _problem(shape, **kw):
    from phasefield5d_b200 import workload as W
    cfg = W.batched_configs(1, seed=5, steps=40)[0]
    cfg.shape, cfg.system_dim = shape, len(shape)
    cfg.adaptive = kw.pop("adaptive", True)
    return dataclasses.replace(W.build_batched_problems([cfg])[0][0], **kw)


def _solve(form, prob, oob_interval):
    from phasefield5d_b200.batch import BatchStepper
    from phasefield5d_b200.stepper import Stepper
    if form == "batch":
        b = BatchStepper([prob], autotune=False, oob_interval=oob_interval)
        return b, lambda: b.states()[0], lambda: b.field(0).cpu().numpy()
    st = Stepper.from_problem(prob, precision=form, autotune=False, oob_interval=oob_interval)
    return st, st.state, lambda: st.field().cpu().numpy()


@pytest.mark.parametrize("form,shape", [("batch", (2048, 2048)), ("fp64", (1024, 1024)),
                                        ("fp32c", (1024, 1024))])
def test_halting_update_writes_every_point(torch_cuda, form, shape):
    prob = _problem(shape, adaptive=False, bk=None, lvec=None)
    st, state, field = _solve(form, prob, 0)
    st.advance(1)
    xdotmax = state()["xdotmax"]
    st.close()
    # one step of a time step that carries most points far out of bounds
    st, state, field = _solve(form, dataclasses.replace(prob, dt0=100.0 / xdotmax), 1)
    st.advance(1)
    s, x = state(), field()
    assert s["halted"] and s["step"] == 1
    moved = (np.abs(x - prob.X_init) > 1e-6).any(axis=-1)
    assert moved.all(), f"{(~moved).sum()} of {moved.size} points were left out"
    st.advance(3)
    after = state()
    assert (after["step"], after["dt"], after["time"]) == (1, s["dt"], s["time"])
    assert np.array_equal(field(), x)
    st.close()


@pytest.mark.parametrize("form,shape", [("fp64", (300, 512)), ("fp32c", (300, 512)),
                                        ("batch", (300, 512)), ("fp64", (24, 40, 50)),
                                        ("fp32c", (24, 40, 50)), ("fp64", (20000,)),
                                        ("fp64", (1000,)), ("fp32c", (1000,)), ("batch", (5000,))])
def test_non_finite_points_end_the_loop_before_the_update(torch_cuda, form, shape):
    prob = _problem(shape, bk=None, lvec=None)
    X = prob.X_init.copy()
    X.reshape(-1, 4)[::397, 1] = np.nan
    prob = dataclasses.replace(prob, X_init=X)
    st, state, field = _solve(form, prob, 0)
    variants = st.n_variants if len(shape) > 1 else 1
    st.close()
    for v in range(variants):
        st, state, field = _solve(form, prob, 0)
        st.set_variant(v)
        before = field()
        st.advance(3)
        s = state()
        assert s["halted"] and s["nn_nonfinite"] and s["step"] == 0 and s["time"] == 0.0, (v, s)
        assert np.array_equal(field(), before, equal_nan=True), v
        st.close()
