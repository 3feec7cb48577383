"""out_of_bounds' kept scratch: many threads on their own streams at once, more
than are kept, each with its own field -- every call answers for its own field."""
import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [1, 20])
def test_calls_on_many_streams_keep_apart(threads):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from phasefield5d_b200 import _lib
    L = _lib.load()
    fields = [torch.full((5000 + 100 * i, 4), 0.01 * (i + 1), dtype=torch.float64, device="cuda")
              for i in range(threads)]
    torch.cuda.synchronize()
    wrong = []

    def work(i):
        stream = torch.cuda.Stream()
        out = (ctypes.c_double * 5)()
        v = 0.01 * (i + 1)
        want = [0.0, ((v + v) + v) + v, ((v + v) + v) + v, v, v]
        for _ in range(25):
            st = L.pf5d_oob_stats(_lib.ptr(fields[i]), fields[i].shape[0], 4, out,
                                  ctypes.c_void_p(stream.cuda_stream))
            if st != 0 or not np.array_equal(list(out), want):
                wrong.append((i, st, list(out)))

    pool = [threading.Thread(target=work, args=(i,)) for i in range(threads)]
    for t in pool:
        t.start()
    for t in pool:
        t.join()
    assert not wrong, wrong[:3]
