"""The batched form's split variants against its first fused one, bit for bit
(mu/M and then faces form every value with the fused kernels' routines in their
order; the FFT plans are the same): sides below, at and past a warp's 30 and 32
columns, the 8, 16 and 32 rows of the kernels' tiles, 1D solves around a tile of
128 points, and lanes without any 2D solve."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = {
    "ragged": [(127,), (3, 5), (129,), (8, 30), (1,), (17, 31), (33, 62), (31, 33)],
    "flat": [(64, 2), (1, 40), (2, 64), (65, 61)],
    "one": [(35, 97)],
    "no_2d": [(130,), (257,)],
}


@pytest.mark.parametrize("kind", list(SHAPES))
def test_split_variants_equal_fused(kind):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from phasefield5d_b200 import workload as W
    from phasefield5d_b200.batch import BatchStepper
    shapes = SHAPES[kind]
    cfgs = W.batched_configs(len(shapes), seed=5, steps=40)
    for c, sh in zip(cfgs, shapes):
        c.shape = sh
        c.system_dim = len(sh)
    probs, _ = W.build_batched_problems(cfgs)
    if kind == "ragged":
        # elastic off for its 2D solves: the batched plans refuse the group after
        # one with an odd number of points (its field is not 8-byte aligned)
        probs = [dataclasses.replace(p, bk=None) if p.dim == 2 else p for p in probs]
    want = None
    for v in range(BatchStepper(probs[:1], autotune=False).n_variants):
        b = BatchStepper(probs, autotune=False)
        b.set_variant(v)
        b.advance(11)
        got = [b.field(i).cpu().numpy() for i in range(len(shapes))]
        states = [(s["dt"], s["time"], s["xdotmax"], s["step"], s["flags"]) for s in b.states()]
        b.close()
        if want is None:
            want = got, states
            assert all(np.isfinite(f).all() for f in got)
        assert states == want[1], v
        for f, r in zip(got, want[0]):
            assert np.array_equal(f, r), v
