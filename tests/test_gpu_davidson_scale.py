"""Davidson roots of a Hamiltonian far from unit scale: all integrals times a power of two, so that the
Hamiltonian's roots are the unscaled ones times it.  The small dense problem of a step takes its
rotation angles in FP32, whose range these norms leave.  Roots within 1e-11 of the largest
diagonal element's scale (residual norms of 1e-13 of it); where the scale is below the solver's
absolute tolerance, the start block's Ritz values stand, finite and of that size."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("realonly", [False, True])
@pytest.mark.parametrize("power", [-180, -140, 100, 140, 300])
def test_scaled_hamiltonian(gpu_lib, realonly, power):
    from dirac_caspt2_gb300 import api, synth
    s = api.SystemInput.from_synth(synth.make_system(synth.SynthConfig(2, 10, 4, 5, seed=31, realonly=realonly)))
    s = dataclasses.replace(s, ecore=0.0)
    f = 2.0 ** power
    t = dataclasses.replace(s, h=np.asarray(s.h) * f, rec_val=np.asarray(s.rec_val) * f)
    with api.Caspt2Session(0) as ses:
        ses.set_casci_solver("davidson")
        ses.set_system(s)
        e0, _ = ses.casci(3)
        ses.set_system(t)
        e1, _ = ses.casci(3)
    e0, e1 = np.asarray(e0), np.asarray(e1) / f
    scale = np.abs(e0).max()
    assert np.isfinite(e1).all()
    if power > 0:
        assert np.abs(e1 - e0).max() <= 1e-11 * scale
    else:
        assert np.abs(e1).max() <= 2 * scale
