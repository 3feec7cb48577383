"""The drop-in functions on shapes and layouts around their kernels' tiles:
sides below, at and past a warp's 30 or 32 columns and a march's chunk, mu and M
as parts of rows of nine and apart, arrays that are not 16-byte aligned --
against the oracle, bit for bit (the elastic term: within the transforms'
rounding)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1,), (5,), (30,), (31,), (121,), (3, 4), (17, 30), (16, 61), (65, 33), (2, 3, 4), (5, 4, 31),
          (9, 7, 61), (18, 5, 30)]


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _shifted(torch, a, shift):
    """A CUDA copy of a, `shift` doubles into its buffer."""
    buf = torch.empty(a.size + shift, dtype=torch.float64, device="cuda")
    view = buf[shift:].view(*a.shape)
    view.copy_(torch.from_numpy(np.ascontiguousarray(a)))
    return view


def _inputs(shape, seed=4):
    rng = np.random.default_rng(seed)
    X = rng.uniform(0.02, 0.23, size=(*shape, 4))
    rows = np.concatenate([rng.normal(0.0, 1e4, size=(*shape, 4)),
                           np.exp(rng.normal(-30.0, 0.5, size=(*shape, 5)))], axis=-1)
    return X, rows


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("layout,shift", [("rows", 0), ("rows", 1), ("rows", 2), ("apart", 0)])
def test_divergence_equals_oracle(torch_cuda, shape, layout, shift):
    from oracle import oracle as O
    from phasefield5d_b200.solver.fluxes import get_divergence_from_mu_function
    X, rows = _inputs(shape)
    want = np.empty_like(X)
    O.get_divergence_from_mu_function(len(shape))(X, np.ascontiguousarray(rows[..., 4:]),
                                                  np.ascontiguousarray(rows[..., :4]), 1e9, want)
    r = _shifted(torch_cuda, rows, shift)
    mu, M = r[..., :4], r[..., 4:]
    if layout == "apart":
        mu, M = mu.contiguous(), M.contiguous()
    out = _shifted(torch_cuda, np.zeros_like(X), shift)
    get_divergence_from_mu_function(len(shape))(_shifted(torch_cuda, X, shift), M, mu, 1e9, out)
    assert np.array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("shift", [0, 1, 2])
def test_laplacian_equals_oracle(torch_cuda, shape, shift):
    from oracle import oracle as O
    from phasefield5d_b200.solver.operators import calculate_laplacian
    X, _ = _inputs(shape)
    got = calculate_laplacian(_shifted(torch_cuda, X, shift), 2e-10)
    assert np.array_equal(got.cpu().numpy(), O.calculate_laplacian(X, 2e-10))


@pytest.mark.parametrize("shape", [(8, 3), (16, 33), (64, 5, 6), (30, 7)])
def test_elastic_update_matches_oracle(torch_cuda, shape):
    from oracle import oracle as O
    from phasefield5d_b200 import workload as W
    from phasefield5d_b200.solver.elastic import make_elastic_updater
    cfg = W.SolveConfig(system_dim=len(shape), initial_composition=(0.1, 0.2, 0.2, 0.25),
                        resolution=0.05, kappa_value=5e-16, mw=4, ppw=16, shape=shape, n_k=500)
    prob = W.build_problem(cfg)
    X, rows = _inputs(shape)
    want = np.ascontiguousarray(rows[..., :4])
    O.make_elastic_updater(prob.X0, prob.lvec, prob.bk, (*shape, 4))(want, X)
    r = torch_cuda.from_numpy(rows).cuda()
    make_elastic_updater(cfg, prob.Lambda, prob.bk, (*shape, 4))(r[..., :4],
                                                                torch_cuda.from_numpy(X).cuda())
    added = np.abs(want - rows[..., :4]).max()
    assert added > 0
    assert np.abs(r[..., :4].cpu().numpy() - want).max() <= 1e-12 * (added + 1e4)
    assert np.array_equal(r[..., 4:].cpu().numpy(), rows[..., 4:])
