"""Second-order sums against the oracle at the sizes where their kernels change form: G with 4350
outer indices of 4 (a thread each), with 10 active spinors (a second group of active indices),
E and F with short sums, and one active spinor pair.  Every e2 within 1e-9 Eh, every sumc2
within 1e-9."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(10, 4, 30, 2), (4, 10, 6, 2), (6, 2, 12, 2)])
def test_energy_sums_match_oracle(gpu_lib, dims):
    from conftest import oracle_system
    from dirac_caspt2_gb300 import api, synth
    from oracle import caspt2_oracle as O
    s = api.SystemInput.from_synth(synth.make_system(synth.SynthConfig(*dims, seed=53)))
    with api.Caspt2Session(0) as ses:
        r = ses.solve(s)
    ref = O.run(oracle_system(s))
    for k in api.SUBSPACES:
        assert abs(r.e2[k] - ref.e2[k]) <= 1e-9, k
        assert abs(r.sumc2[k] - ref.sumc2[k]) <= 1e-9, k
