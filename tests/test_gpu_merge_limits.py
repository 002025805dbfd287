"""Merged Householder reductions keep each context's own wait limit, whichever context leads the
joint launch: with 1 ns in one of two contexts that one's waits run out (DCG_E_NUMERIC) and the
other gets the bits of its matrix alone.  The waits are bounded and the kernel leaves by itself."""
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _herm(n, seed):
    rng = np.random.default_rng(seed)
    X = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
    return X + X.conj().T


@pytest.mark.parametrize("short_leads", [True, False])
def test_limit_of_each_context(gpu_lib, monkeypatch, short_leads):
    from dirac_caspt2_gb300 import api
    n = 400
    mats = {"short": _herm(n, 1), "plain": _herm(n, 2)}
    alone = {}
    for name, H in mats.items():
        with api.Caspt2Session(0) as ses:
            alone[name] = ses.heev(H, vectors=False)
    monkeypatch.setenv("DCG_MERGE_WINDOW_US", "2000000")
    ses = {name: api.Caspt2Session(0) for name in mats}
    for s in ses.values():
        assert s.lib.dcg_set_merge_reductions(s.h, 1) == 0
    ses["short"].set_wait_limit(1e-9)
    out = {"short": [], "plain": []}

    def run(name):
        try:
            out[name].append(ses[name].heev(mats[name], vectors=False))
        except api.DcgError as e:
            out[name].append(e)

    order = ["short", "plain"] if short_leads else ["plain", "short"]
    m0 = api.merged_reduction_stats(0)
    try:
        for _ in range(3):
            th = [threading.Thread(target=run, args=(name,)) for name in order]
            th[0].start()
            time.sleep(0.2)   # the first one waits for company and leads
            th[1].start()
            for t in th:
                t.join(60)
    finally:
        for s in ses.values():
            s.close()
    assert api.merged_reduction_stats(0)["joint_launches"] - m0["joint_launches"] == 3
    for r in out["plain"]:
        assert not isinstance(r, Exception), r
        assert np.array_equal(r, alone["plain"])
    raised = 0
    for r in out["short"]:   # a wait gives up once a block has polled for longer than the limit
        if isinstance(r, Exception):
            assert r.code == -6 and "timed out" in str(r)
            raised += 1
        else:
            assert np.array_equal(r, alone["short"])
    assert raised > 0
