"""A real-only system runs on real arithmetic; the same integrals declared complex (zero imaginary
parts) run on complex arithmetic: the energies agree to rounding.  A real-only system whose
one-electron integrals do have imaginary parts keeps complex arithmetic.

Tolerance 1e-11 Eh: both paths are FP64 with sums of different order, a few hundred units of
rounding of energies of order 100 Eh (1.4e-14 each)."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solve(s, prec):
    from dirac_caspt2_gb300 import api
    with api.Caspt2Session(0, prec) as ses:
        return ses.solve(s)


def _same(a, b):
    assert np.abs(a.casci_energies - b.casci_energies).max() <= 1e-11
    for k in a.e2:
        assert abs(a.e2[k] - b.e2[k]) <= 1e-11, k
        assert abs(a.sumc2[k] - b.sumc2[k]) <= 1e-11, k
    assert abs(a.total_energy - b.total_energy) <= 1e-11


@pytest.mark.parametrize("dims", [(4, 4, 10, 2), (2, 8, 22, 4), (6, 10, 36, 4), (2, 12, 8, 6)])
@pytest.mark.parametrize("complex_h", [False, True])
def test_real_arithmetic_matches_complex(gpu_lib, dims, complex_h):
    from dirac_caspt2_gb300 import api, synth
    s = api.SystemInput.from_synth(synth.make_system(synth.SynthConfig(*dims, seed=17, realonly=True)))
    if complex_h:
        g = np.random.default_rng(3).normal(size=s.h.shape) * 1e-3
        s = dataclasses.replace(s, h=s.h + 1j * (g - g.T))
    c = dataclasses.replace(s, realonly=False, rec_val=np.asarray(s.rec_val, np.complex128))
    _same(_solve(s, api.DCG_PREC_FP64), _solve(c, api.DCG_PREC_FP64))
