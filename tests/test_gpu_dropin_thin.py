"""The drop-in divergence and Laplacian on fields with a short last axis, whose
points fill few lanes of the tiled kernels: the values on both sides of the
rules that choose a kernel, and the cost per point, which stays that of a field
with full tiles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("layout", ["rows", "apart"])
@pytest.mark.parametrize("shape", [(41, 1), (40, 8), (40, 9), (33, 13), (33, 14), (9, 4, 15), (9, 4, 22),
                                   (5, 8, 31), (7, 1, 30), (7, 2, 24), (7, 3, 27), (6, 5, 30), (6, 6, 30),
                                   (3, 7, 64), (4, 16, 128), (23, 24, 60), (41, 27, 30)])
def test_values_on_both_sides_of_the_rules(torch_cuda, shape, layout):
    from oracle import oracle as O
    from phasefield5d_b200.solver.fluxes import get_divergence_from_mu_function
    from phasefield5d_b200.solver.operators import calculate_laplacian
    rng = np.random.default_rng(6)
    X = rng.uniform(0.02, 0.23, size=(*shape, 4))
    rows = np.concatenate([rng.normal(0.0, 1e4, size=(*shape, 4)),
                           np.exp(rng.normal(-30.0, 0.5, size=(*shape, 5)))], axis=-1)
    want = np.empty_like(X)
    O.get_divergence_from_mu_function(len(shape))(X, np.ascontiguousarray(rows[..., 4:]),
                                                  np.ascontiguousarray(rows[..., :4]), 1e9, want)
    x, r = torch_cuda.from_numpy(X).cuda(), torch_cuda.from_numpy(rows).cuda()
    mu, M = r[..., :4], r[..., 4:]
    if layout == "apart":
        mu, M = mu.contiguous(), M.contiguous()
    out = torch_cuda.empty_like(x)
    get_divergence_from_mu_function(len(shape))(x, M, mu, 1e9, out)
    assert np.array_equal(out.cpu().numpy(), want)
    got = calculate_laplacian(x, 2e-10)
    assert np.array_equal(got.cpu().numpy(), O.calculate_laplacian(X, 2e-10))


def _us(torch, call, reps=20):
    best = float("inf")
    for _ in range(8):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        torch.cuda._sleep(2_000_000)         # the calls are queued before they run
        a.record()
        for _ in range(reps):
            call()
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) * 1e3 / reps)
    return best


@pytest.mark.parametrize("what", ["divergence_rows", "divergence_apart", "laplacian"])
def test_thin_fields_cost_no_more_per_point(torch_cuda, what):
    """A point per thread costs about the same for any shape: 1.3 times (rows),
    2.0 times (apart) and 1.9 times (Laplacian) what a point of a 128^3 field
    costs in its tiled kernel.  Half as much again is allowed; tiles with few
    full lanes cost 4 to 14 times as much."""
    torch = torch_cuda
    from phasefield5d_b200.solver.fluxes import get_divergence_from_mu_function
    from phasefield5d_b200.solver.operators import calculate_laplacian
    per_point = {}
    for shape in [(128, 128, 128), (1_000_000, 1), (500_000, 4), (1024, 512, 2), (60_000, 4, 4),
                  (400_000, 5, 1)]:
        X = torch.full((*shape, 4), 0.2, dtype=torch.float64, device="cuda")
        I = torch.full((*shape, 9), 0.1, dtype=torch.float64, device="cuda")
        out, mu, M = torch.empty_like(X), I[..., :4], I[..., 4:]
        if what == "divergence_apart":
            mu, M = mu.contiguous(), M.contiguous()
        div = get_divergence_from_mu_function(len(shape))
        if what == "laplacian":
            us = _us(torch, lambda: calculate_laplacian(X, 1e-9, out=out))
        else:
            us = _us(torch, lambda: div(X, M, mu, 1e9, out))
        per_point[shape] = us / (X.numel() // 4)
    full = per_point.pop((128, 128, 128))
    allowed = {"divergence_rows": 2.0, "divergence_apart": 3.0, "laplacian": 3.0}[what]
    assert max(per_point.values()) <= allowed * full, (full, per_point)
