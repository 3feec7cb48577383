"""The 1D step loop (one cluster, many steps per launch) against the same steps
launched stage by stage, bit for bit: sizes around a warp, a block's chunk and
the longest solve, every option of a step, and the halts inside a launch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FORMS = ["fp64", "fp32c"]


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _problem(n, elastic=True, adaptive=True):
    from phasefield5d_b200 import workload as W
    cfg = W.SolveConfig(system_dim=1, initial_composition=(0.1, 0.2, 0.2, 0.25), resolution=0.05,
                        kappa_value=5e-16, mw=4, ppw=16, shape=(n,), n_k=500, adaptive=adaptive,
                        include_cubic_anisotropy=elastic, fluctuation=2e-2)
    return W.build_problem(cfg)


def _stepper(prob, precision, X=None, **kw):
    import dataclasses
    from phasefield5d_b200.stepper import Stepper
    if X is not None:
        prob = dataclasses.replace(prob, X_init=X)
    return Stepper.from_problem(prob, precision=precision, **kw)


def _staged(st, n, elastic):
    from phasefield5d_b200 import _lib
    for _ in range(n):
        if elastic:
            st.launch_stage(_lib.STAGE_FFT_FWD)
        st.launch_stage(_lib.STAGE_RATE)
        st.launch_stage(_lib.STAGE_UPDATE)


def _same(a, b, precision, rate=True):
    assert a.state() == b.state()
    assert np.array_equal(a.field().cpu().numpy(), b.field().cpu().numpy(), equal_nan=True)
    if rate and precision == "fp64":
        assert np.array_equal(a.rate().cpu().numpy(), b.rate().cpu().numpy(), equal_nan=True)


@pytest.mark.parametrize("precision", FORMS)
@pytest.mark.parametrize("n", [3, 31, 32, 33, 203, 511, 513, 1280, 7680, 7681, 16384])
def test_loop_equals_stages(torch_cuda, precision, n):
    prob = _problem(n)
    a, b = _stepper(prob, precision), _stepper(prob, precision)
    a.advance(5)
    a.advance(1)
    _staged(b, 6, True)
    _same(a, b, precision)
    a.close()
    b.close()


@pytest.mark.parametrize("precision", FORMS)
@pytest.mark.parametrize("elastic,adaptive,interval", [(False, True, 100), (True, False, 2), (True, True, 0)])
def test_loop_options(torch_cuda, precision, elastic, adaptive, interval):
    prob = _problem(300, elastic, adaptive)
    a, b = (_stepper(prob, precision, oob_interval=interval) for _ in range(2))
    a.advance(7)
    _staged(b, 7, elastic)
    _same(a, b, precision)
    a.close()
    b.close()


@pytest.mark.parametrize("precision", FORMS)
@pytest.mark.parametrize("what", ["far", "soft", "hard", "nan"])
def test_loop_halts_as_stages(torch_cuda, precision, what):
    """Points on the nearest-row fallback, and out-of-bounds values that the
    test inside the launch finds (soft: flagged, hard: halted) or that reach
    the fallback first (NaN)."""
    prob = _problem(700)
    X = prob.X_init.copy()
    X[333] = {"far": [0.3, 0.3, 0.2, 0.15], "soft": [-5e-5, 0.2, 0.2, 0.2],
              "hard": [-5e-3, 0.2, 0.2, 0.2], "nan": [np.nan, 0.2, 0.2, 0.2]}[what]
    runs = []
    for staged in (False, True):
        st = _stepper(prob, precision)
        st.X.copy_(torch_cuda.from_numpy(X))
        st.reset(prob.dt0)
        if what in ("hard", "nan"):
            assert st.state()["halted"]          # reset's own test halts before any step
        (lambda: _staged(st, 150, True) if staged else st.advance(150))()
        runs.append(st)
    _same(*runs, precision, rate=what not in ("hard", "nan"))
    for st in runs:
        st.close()


@pytest.mark.parametrize("precision", FORMS)
def test_loop_stops_inside_a_launch(torch_cuda, precision):
    """A nearest-row distance error and an out-of-bounds halt raised by a later
    step of one launch leave the state the stages leave."""
    prob = _problem(700)
    X = prob.X_init.copy()
    X[100] = [0.3, 0.3, 0.2, 0.15]                # a table row: too far only once it has moved
    runs = []
    for staged in (False, True):
        st = _stepper(prob, precision, X=X, max_nn_dist=1e-6)
        (lambda: _staged(st, 20, True) if staged else st.advance(20))()
        assert st.state()["halted"] and st.state()["nn_far"] and 0 < st.state()["step"] < 20
        runs.append(st)
    _same(*runs, precision)
    for st in runs:
        st.close()
    runs = []
    for staged in (False, True):
        st = _stepper(_problem(700, adaptive=False), precision, oob_interval=5)
        st.reset(3e4 * prob.t_cfl)                # far above the stable step: leaves the simplex
        (lambda: _staged(st, 40, True) if staged else st.advance(40))()
        assert st.state()["halted"] and 0 < st.state()["step"] < 40
        runs.append(st)
    _same(*runs, precision)
    for st in runs:
        st.close()
