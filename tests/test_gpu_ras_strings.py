"""The determinants of a RAS space are put together from their RAS3, RAS2 and RAS1 parts: their
number against a count over all bit strings, and, where the ranges exclude nothing, the roots
of the unrestricted space (the same matrix: 1e-11 Eh)."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (spinors, electrons), (ras1, ras2, ras3), (holes, particles), (least holes, least particles)
CASES = [((8, 4), (4, 4, 0), (2, 0), (0, 0)),      # no RAS3
         ((8, 4), (0, 4, 4), (0, 2), (0, 0)),      # no RAS1
         ((8, 4), (2, 2, 4), (1, 3), (1, 1)),      # least numbers
         ((8, 5), (4, 0, 4), (2, 2), (0, 0)),      # no RAS2
         ((8, 3), (2, 4, 2), (2, 2), (0, 0)),      # nothing excluded
         ((6, 6), (2, 2, 2), (0, 2), (0, 0))]      # every spinor filled


def _system(space, ras, most, least):
    from dirac_caspt2_gb300 import api, synth
    s = api.SystemInput.from_synth(synth.make_system(synth.SynthConfig(2, space[0], 4, space[1], seed=47)))
    s.ras = ras
    s.ras1_max_hole, s.ras3_max_elec = most
    s.min_hole_ras1, s.min_elec_ras3 = least
    return s


@pytest.mark.parametrize("space,ras,most,least", CASES)
def test_ras_strings(gpu_lib, space, ras, most, least):
    from dirac_caspt2_gb300 import api
    na, ne = space
    keep = 0
    for b in range(1 << na):
        if bin(b).count("1") != ne:
            continue
        holes = ras[0] - bin(b & ((1 << ras[0]) - 1)).count("1")
        parts = bin(b >> (ras[0] + ras[1])).count("1")
        keep += (ras[0] == 0 or least[0] <= holes <= most[0]) and (ras[2] == 0 or least[1] <= parts <= most[1])
    with api.Caspt2Session(0) as ses:
        ses.set_system(_system(space, ras, most, least))
        e, n = ses.casci(1)
        assert n == keep
        if keep == math.comb(na, ne):
            ses.set_system(_system(space, (0, 0, 0), (0, 0), (0, 0)))
            full, m = ses.casci(1)
            assert m == n and np.abs(np.asarray(e) - np.asarray(full)).max() <= 1e-11
