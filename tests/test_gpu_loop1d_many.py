"""Solves of several lengths at once: a step loop launched after shorter solves
were created runs as it does alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
def test_longer_solve_runs_after_shorter_ones_were_created(precision):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from phasefield5d_b200 import workload as W
    from phasefield5d_b200.stepper import Stepper
    probs = [W.build_problem(W.SolveConfig(
        system_dim=1, initial_composition=(0.1, 0.2, 0.2, 0.25), resolution=0.05, kappa_value=5e-16,
        mw=4, ppw=16, shape=(n,), n_k=500, fluctuation=2e-2)) for n in (16384, 4112, 203)]
    alone = []
    for p in probs:
        st = Stepper.from_problem(p, precision=precision)
        st.advance(7)
        alone.append(st.field().cpu().numpy())
        st.close()
    together = [Stepper.from_problem(p, precision=precision) for p in probs]
    for st in together:
        st.advance(7)
    for st, want in zip(together, alone):
        assert np.array_equal(st.field().cpu().numpy(), want)
        st.close()
