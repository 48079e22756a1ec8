"""A new context's buffers are cleared before anything that its streams do: a field set while
another thread keeps the default stream busy keeps its values."""
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_first_upload_is_not_cleared_late(gb):
    a = torch.randn(1024, 1024, device="cuda", dtype=torch.float64)
    b = a @ a
    torch.cuda.synchronize()
    stop = threading.Event()

    def busy():
        pending = []
        while not stop.is_set():  # a few milliseconds queued on the default stream at any time
            torch.matmul(a, a, out=b)
            e = torch.cuda.Event()
            e.record()
            pending.append(e)
            if len(pending) > 4:
                pending.pop(0).synchronize()

    t = threading.Thread(target=busy)
    t.start()
    try:
        phi = np.random.default_rng(3).standard_normal((33 + 4, 40 + 4))
        for _ in range(10):
            c = gb.Context(40, 33)
            c.set(gb.FIELD_PHI, phi)
            torch.cuda.synchronize()
            got = c.get(gb.FIELD_PHI)
            c.close()
            np.testing.assert_array_equal(got, phi)
    finally:
        stop.set()
        t.join()
