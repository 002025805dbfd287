"""Davidson on nearly degenerate active levels (within 1e-4), where restarts every few steps can stall:
two roots of 8,008 determinants converge within the solver's steps, and agree with the lowest two
of four (each within its residual norm, 1e-13 of a largest diagonal element of order 100, of an
eigenvalue: 2e-11 between the two)."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("realonly", [False, True])
@pytest.mark.parametrize("scale", [1.0, 0.05])   # of the couplings and the interaction
def test_near_degenerate_levels(gpu_lib, realonly, scale):
    from dirac_caspt2_gb300 import api, synth
    s = api.SystemInput.from_synth(synth.make_system(synth.SynthConfig(2, 16, 4, 6, seed=7, realonly=realonly)))
    h = np.array(s.h) * scale
    level = np.concatenate([np.full(2, -20.0), -1.0 + 1e-4 * np.random.default_rng(3).normal(size=16),
                            np.full(len(h) - 18, 5.0)])
    np.fill_diagonal(h, level)
    s = dataclasses.replace(s, h=h, rec_val=np.asarray(s.rec_val) * scale)
    with api.Caspt2Session(0) as ses:
        ses.set_casci_solver("davidson")
        ses.set_system(s)
        e2, n = ses.casci(2)
        e4, _ = ses.casci(4)
    assert n == 8008
    assert np.abs(np.asarray(e2) - np.asarray(e4)[:2]).max() <= 2e-11
