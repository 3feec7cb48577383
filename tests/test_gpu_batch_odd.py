"""Batches of elastic 2D solves with odd numbers of points: the shape group after
one of them starts at an aligned place, every variant gives the same bits, and
each solve follows its plain-FP64 run."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(127,), (33, 31), (8, 30), (17, 31), (1,), (31, 33), (3, 5), (62, 33), (33, 31)]


def test_odd_shapes_with_elasticity():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from phasefield5d_b200 import workload as W
    from phasefield5d_b200.batch import BatchStepper
    from phasefield5d_b200.stepper import Stepper
    cfgs = W.batched_configs(len(SHAPES), seed=5, steps=40)
    for c, sh in zip(cfgs, SHAPES):
        c.shape = sh
        c.system_dim = len(sh)
    probs, _ = W.build_batched_problems(cfgs)
    assert all(p.bk is not None for p in probs)
    want = None
    for v in range(BatchStepper(probs[:1], autotune=False).n_variants):
        b = BatchStepper(probs, autotune=False)
        b.set_variant(v)
        b.advance(20)
        got = [b.field(i).cpu().numpy() for i in range(len(probs))]
        b.close()
        want = want or got
        assert all(np.array_equal(g, w) for g, w in zip(got, want)), v
    for p, X in zip(probs, want):
        st = Stepper.from_problem(p)
        st.run(20)
        ref = st.X.cpu().numpy()
        st.close()
        assert np.max(np.abs(X - ref)) <= 1e-6 * np.max(np.abs(ref)), p.shape
