"""The split variants' mu/M buffer (40 bytes per point) of a batch: held only
while one of them runs, and back for the next use of the memory otherwise.  The
sizes are far above the allocator's granularity."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_batch_holds_the_split_buffer_only_for_split_variants():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from phasefield5d_b200 import workload as W
    from phasefield5d_b200.batch import BatchStepper
    shapes = [(1024, 1024), (1023, 1023)]
    cfgs = W.batched_configs(len(shapes), seed=5, steps=40)
    for c, sh in zip(cfgs, shapes):
        c.shape = sh
        c.system_dim = 2
    probs, _ = W.build_batched_problems(cfgs)
    need = 40 * sum(p.n_points for p in probs)

    def held():
        torch.cuda.synchronize()
        free, total = torch.cuda.mem_get_info()
        return total - free

    b = BatchStepper(probs, autotune=False)
    b.advance(2)
    fused = held()
    b.set_variant(b.n_variants - 1)          # split
    b.advance(2)
    assert held() - fused >= need
    b.set_variant(0)
    b.advance(2)
    assert held() - fused < need // 4
    got = [b.field(i).cpu().numpy() for i in range(len(shapes))]
    b.close()
    b = BatchStepper(probs, autotune=False)
    b.advance(6)
    for i, f in enumerate(got):
        assert np.array_equal(f, b.field(i).cpu().numpy())
    b.close()


def test_variant_changes_wait_for_the_steps_before():
    """Steps enqueued on the batch's own stream run with the variant they were
    enqueued with, also where the next one is chosen before they have run."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from phasefield5d_b200 import workload as W
    from phasefield5d_b200.batch import BatchStepper
    cfgs = W.batched_configs(2, seed=5, steps=40)
    for c, sh in zip(cfgs, [(256, 250), (1024,)]):
        c.shape, c.system_dim = sh, len(sh)
    probs, _ = W.build_batched_problems(cfgs)
    got = []
    for wait in (True, False):
        own = torch.cuda.Stream()
        with torch.cuda.stream(own):
            b = BatchStepper(probs, stream=own, autotune=False)
        for v in (b.n_variants - 1, 0, b.n_variants - 2, 3):
            b.set_variant(v)
            b.advance(200)
            if wait:
                torch.cuda.synchronize()
        got.append([b.field(i).cpu().numpy() for i in range(2)])
        b.close()
    for a, c in zip(*got):
        assert np.array_equal(a, c)
