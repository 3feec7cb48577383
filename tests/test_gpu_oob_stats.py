"""Out-of-bounds statistics against numpy: sizes around a warp, a block and a
full grid, rows that are not four components or not 16-byte aligned, and
non-finite values (which leave their row's sum out)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("ncomp,shift", [(4, 0), (4, 1), (3, 0), (5, 0)])
@pytest.mark.parametrize("npts", [1, 31, 257, 303105])
@pytest.mark.parametrize("bad", [False, True])
def test_oob_stats_equal_numpy(torch_cuda, ncomp, shift, npts, bad):
    from phasefield5d_b200 import _lib
    rng = np.random.default_rng(npts + ncomp)
    x = rng.uniform(-0.2, 0.5, size=(npts, ncomp))
    if bad:
        x[rng.integers(0, npts, size=3), rng.integers(0, ncomp, size=3)] = [np.nan, np.inf, -np.inf]
    buf = torch_cuda.empty(npts * ncomp + shift, dtype=torch_cuda.float64, device="cuda")
    dev = buf[shift:]
    dev.copy_(torch_cuda.from_numpy(x.reshape(-1)))
    ptr, got = _lib.f64_array([0.0] * 5)
    _lib.check(_lib.load().pf5d_oob_stats(_lib.ptr(dev), npts, ncomp, ptr, _lib.stream_handle()))
    ok = np.isfinite(x)
    rows = ok.all(axis=1)
    sums = np.zeros(npts)
    for c in range(ncomp):
        sums = sums + x[:, c]
    assert got[0] == np.count_nonzero(~ok)
    if rows.any():
        assert (got[1], got[2]) == (sums[rows].max(), sums[rows].min())
    if ok.any():
        assert (got[3], got[4]) == (x[ok].max(), x[ok].min())
