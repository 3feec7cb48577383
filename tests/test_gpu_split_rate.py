"""The split rate stage (every point's mu/M once, then the faces) against the
fused one, bit for bit, where its tiles can go wrong: sides below, at and just
past the tiles' sides, and fields that fill the work items in every way (one
cell, the cells around a node, cells all over the table with hash collisions,
points outside the linear region), for tables with and without vector-aligned
nodes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _field(kind, shape, rng):
    x = np.broadcast_to(np.array([0.1, 0.2, 0.2, 0.25]), (*shape, 4))
    if kind == "cell":
        return x + 0.02 + rng.uniform(-1e-3, 1e-3, size=x.shape)
    if kind == "node":
        return x + rng.uniform(-1e-3, 1e-3, size=x.shape)
    return rng.dirichlet(np.full(5, 3.0), size=shape)[..., 1:]      # all over, some far


def _run(prob, X, variant, table, precision="fp64"):
    """Field and dX/dt after two steps (the precision form's dX/dt is float32
    and not compared)."""
    from phasefield5d_b200.stepper import Stepper
    st = Stepper(grid=prob.grid, resolution=prob.cfg.resolution, node_coord=prob.node_coord, X=X,
                 X0=prob.X0, kappa=prob.kappa, dx=prob.dx, lvec=prob.lvec, bk=prob.bk,
                 ctld=prob.ctld, t_cfl=prob.t_cfl, dt=1e-3 * prob.t_cfl, autotune=False, table=table,
                 precision=precision)
    st.set_variant(variant)
    st.run(2)
    state = st.state()
    out = (st.field().cpu().numpy(),
           st.rate().cpu().numpy() if precision == "fp64" else np.array([state["xdotmax"]]))
    st.close()
    return out


def _split_variants(prob, precision="fp64"):
    from phasefield5d_b200.stepper import Stepper
    st = Stepper.from_problem(prob, autotune=False, precision=precision)
    names = []
    for v in range(st.n_variants):
        st.set_variant(v)
        names.append(st.rate_kernels)
    st.close()
    return [v for v, n in enumerate(names) if n.startswith(("k_chem", "k32_chem"))]


@pytest.mark.parametrize("kind", ["cell", "node", "spread"])
@pytest.mark.parametrize("shape", [(3, 5), (16, 32), (17, 33), (31, 63), (50, 130), (4, 4, 32),
                                   (3, 5, 33), (5, 9, 65), (9, 16, 31), (2, 3, 4)])
def test_split_rate_bitwise_equals_fused(torch_cuda, shape, kind):
    from phasefield5d_b200 import workload as W
    cfg = W.SolveConfig(system_dim=len(shape), initial_composition=(0.1, 0.2, 0.2, 0.25),
                        resolution=0.05, kappa_value=5e-16, mw=4, ppw=16, shape=shape, n_k=500)
    prob = W.build_problem(cfg)
    X = _field(kind, shape, np.random.default_rng(3))
    table9 = torch_cuda.from_numpy(np.ascontiguousarray(prob.grid)).cuda()
    ref = _run(prob, X, 0, None)
    assert np.isfinite(ref[1]).all() and np.abs(ref[1]).max() > 0
    for v in _split_variants(prob):
        for table in (None, table9):
            got = _run(prob, X, v, table)
            assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1]), (v, table is None)


@pytest.mark.parametrize("kind", ["cell", "node", "spread"])
@pytest.mark.parametrize("shape", [(3, 5), (16, 32), (17, 33), (50, 130), (4, 4, 32), (3, 5, 33),
                                   (5, 9, 65), (9, 17, 31), (2, 3, 4)])
def test_split_rate_fp32c_bitwise_equals_fused(torch_cuda, shape, kind):
    from phasefield5d_b200 import workload as W
    cfg = W.SolveConfig(system_dim=len(shape), initial_composition=(0.1, 0.2, 0.2, 0.25),
                        resolution=0.05, kappa_value=5e-16, mw=4, ppw=16, shape=shape, n_k=500)
    prob = W.build_problem(cfg)
    X = _field(kind, shape, np.random.default_rng(3))
    ref = _run(prob, X, 0, None, "fp32c")
    assert np.isfinite(ref[0]).all() and ref[1].max() > 0
    for v in _split_variants(prob, "fp32c"):
        got = _run(prob, X, v, None, "fp32c")
        assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1]), v
