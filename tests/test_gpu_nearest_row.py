"""The nearest-row fallback where its rounded-node answer and its scan meet:
exact ties, points one rounding away from a tie, points whose rounded node
lies past the simplex face, and points outside the table, against a brute
force over all rows (first row in lexicographic node order among exactly
equal distances, the distance summed in axis order)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _brute(x, rows):
    out = np.empty(len(x), dtype=np.int64)
    for i in range(0, len(x), 256):
        d = x[i:i + 256, None, :] - rows[None, :, :4]
        e = d[..., 0] * d[..., 0]
        for a in (1, 2, 3):
            e = e + d[..., a] * d[..., a]
        out[i:i + 256] = np.argmin(e, axis=1)
    return out


def _points(kind, res, rng):
    n = int(round(1.0 / res))
    if kind in ("tie", "near_tie"):
        # nodes and cell midpoints mixed per axis, sums past the linear region
        k = rng.integers(0, 2 * n, size=(60000, 4))
        k = k[(k.sum(axis=1) > 2 * (n - 4)) & (k.sum(axis=1) <= 2 * n)][:600]
        x = k * (0.5 * res)
        if kind == "near_tie":
            x = np.nextafter(x, x + rng.choice([-1.0, 1.0], size=x.shape))
        return x
    if kind == "face":
        x = rng.dirichlet(np.ones(5), size=600)
        x[:, 0] *= rng.uniform(0.0, 2.0 * res, size=600)
        return (x / x.sum(axis=1, keepdims=True))[:, 1:]
    return rng.uniform(-0.1, 1.2, size=(600, 4))


@pytest.mark.parametrize("res", [0.05, 0.025])
@pytest.mark.parametrize("kind", ["tie", "near_tie", "face", "outside"])
def test_nearest_row_equals_brute_force(torch_cuda, kind, res):
    from phasefield5d_b200 import workload as W
    from phasefield5d_b200.solver.interpolation import interpolator_nb
    from phasefield5d_b200.solver.table import build_4d_grid, build_calphad_kdtree
    rows = W.make_table(res, 873.0, 4).data
    _, grid = build_4d_grid(rows, res)
    tree, vals = build_calphad_kdtree(rows)
    x = _points(kind, res, np.random.default_rng(11))
    out = np.empty((len(x), 9))
    mask = np.empty(len(x), dtype=np.bool_)
    interpolator_nb(x, grid, res, tree, vals, out=out, mask_buffer=mask)
    bad = ~mask
    assert bad.sum() > 200
    assert np.array_equal(out[bad], vals[_brute(x[bad], rows)])


def test_finite_point_beyond_every_distance_still_raises(torch_cuda, small_table):
    """Squared distances that overflow leave no nearest row."""
    from phasefield5d_b200.solver.interpolation import interpolator_nb
    t = small_table
    with pytest.raises(RuntimeError):
        interpolator_nb(np.array([[1e200, 0.1, 0.1, 0.1]]), t["grid"], t["resolution"], t["tree"],
                        t["vals"])
