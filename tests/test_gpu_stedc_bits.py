"""The same tridiagonal gives the same bits every time, alone and with other streams busy: spectra
whose deflation has many neighbouring runs of close poles."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(kind, n):
    if kind == "wilkinson":
        return np.abs(np.arange(n) - (n - 1) / 2.0), np.ones(n - 1)
    d = np.abs((np.arange(n) % 21) - 10.0)
    e = np.ones(n - 1)
    e[20::21] = 1e-9
    return d, e


@pytest.mark.parametrize("kind", ["glued", "wilkinson"])
def test_same_bits_every_time(gpu_lib, kind):
    from dirac_caspt2_gb300 import api
    d, e = _matrix(kind, 700)
    with api.Caspt2Session(0) as ses, api.Caspt2Session(0) as other:
        w0, z0 = ses.stedc(d, e)
        stop = threading.Event()

        def busy():
            rng = np.random.default_rng(1)
            d2, e2 = rng.normal(size=500), rng.normal(size=499)
            while not stop.is_set():
                other.stedc(d2, e2)

        for alone in (True, False):
            th = None if alone else threading.Thread(target=busy)
            if th:
                th.start()
            try:
                for _ in range(25):
                    w, z = ses.stedc(d, e)
                    assert np.array_equal(w, w0) and np.array_equal(z, z0)
            finally:
                stop.set()
                if th:
                    th.join()
