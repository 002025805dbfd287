"""Davidson on determinant spaces of more than one chunk of rows (1,024), real and complex, CAS and
RAS, against the dense solver on the same Hamiltonian: the requested roots within 1e-11 Eh
(residual norms of 1e-13 give energy errors of their square; the dense solver's own error is a few
units of rounding of energies of order 100 Eh)."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,ras,ndet", [
    ((2, 14, 4, 4), None, 1001), ((2, 14, 4, 5), None, 2002),
    ((2, 14, 4, 6), ((4, 6, 4), 2, 2), 1960),
])
@pytest.mark.parametrize("realonly", [False, True])
@pytest.mark.parametrize("nroot", [1, 4])
def test_roots_match_dense(gpu_lib, dims, ras, ndet, realonly, nroot):
    from dirac_caspt2_gb300 import api, synth
    s = api.SystemInput.from_synth(synth.make_system(synth.SynthConfig(*dims, seed=29, realonly=realonly)))
    if ras:
        s = dataclasses.replace(s, ras=ras[0], ras1_max_hole=ras[1], ras3_max_elec=ras[2])
    with api.Caspt2Session(0) as ses:
        ses.set_system(s)
        ses.set_casci_solver("dense")
        e0, n0 = ses.casci(nroot)
        ses.set_casci_solver("davidson")
        e1, n1 = ses.casci(nroot)
        assert ses.casci_iterations() > 0
    assert n0 == n1
    if ras is None:
        assert n1 == ndet
    assert n1 > 1000
    assert np.abs(np.asarray(e0) - np.asarray(e1)).max() <= 1e-11
