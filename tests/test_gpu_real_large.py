"""Real arithmetic where its kernels change form: dense CI matrices of real systems on both sides of
1,024 rows (columns in shared memory in pieces, columns in global memory, blocked
back-transformation), densities and metrics of 14 active spinors, and split precision.

Vectors: the span of the dense solver's (degenerate roots together) against Davidson's (residual 1e-13
of the largest diagonal element, of order 100): the angle is at most residual / gap, 4e-11 / gap with
both solvers' errors.  Energies and
second-order terms of the same integrals declared complex: 1e-11 Eh in FP64 (sums of another order of
energies of order 100 Eh); 1e-9 on the split path, whose products carry 2^-36 of their operands."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _real(dims, seed):
    from dirac_caspt2_gb300 import api, synth
    return api.SystemInput.from_synth(synth.make_system(synth.SynthConfig(*dims, seed=seed, realonly=True)))


@pytest.mark.parametrize("dims,ndet", [((2, 14, 4, 4), 1001), ((2, 20, 4, 3), 1140), ((2, 14, 4, 5), 2002)])
def test_dense_vectors_match_davidson(gpu_lib, dims, ndet):
    from dirac_caspt2_gb300 import api
    s = _real(dims, 61)
    nroot = 6
    with api.Caspt2Session(0) as ses:
        ses.set_system(s)
        ses.set_casci_solver("dense")
        e0, n0, c0 = ses.casci(nroot, want_ci=True)
        ses.set_casci_solver("davidson")
        e1, n1, c1 = ses.casci(nroot, want_ci=True)
    assert n0 == n1 == ndet
    e0, e1 = np.asarray(e0), np.asarray(e1)
    assert np.abs(e0[:nroot] - e1[:nroot]).max() <= 1e-11
    assert np.abs(c0.imag).max() == 0.0
    V = c0[:, :nroot]
    assert np.abs(V.conj().T @ V - np.eye(nroot)).max() <= 20 * ndet * 2.0 ** -53
    first = 0   # clusters of degenerate roots: the spans agree (the last cluster may be cut off)
    checked = 0
    for r in range(1, nroot):
        gap = e1[r] - e1[r - 1]
        if gap < 1e-6:
            continue
        D = c1[:, first:r]
        out = V[:, first:r] - D @ (D.conj().T @ V[:, first:r])
        assert np.linalg.norm(out, 2) <= 4e-11 / min(gap, e1[first] - e1[first - 1] if first else gap)
        first = r
        checked += 1
    assert checked


@pytest.mark.parametrize("dims", [(2, 14, 6, 4), (12, 8, 60, 4)])
@pytest.mark.parametrize("prec", ["fp64", "split"])
def test_solve_matches_complex(gpu_lib, dims, prec):
    from dirac_caspt2_gb300 import api
    s = _real(dims, 67)
    c = dataclasses.replace(s, realonly=False, rec_val=np.asarray(s.rec_val, np.complex128))
    out = []
    for x in (s, c):
        with api.Caspt2Session(0, api.DCG_PREC_FP64 if prec == "fp64" else api.DCG_PREC_SPLIT) as ses:
            out.append(ses.solve(x))
    tol = 1e-11 if prec == "fp64" else 1e-9
    a, b = out
    assert np.abs(a.casci_energies - b.casci_energies).max() <= 1e-11
    for k in a.e2:
        assert abs(a.e2[k] - b.e2[k]) <= tol, k
        assert abs(a.sumc2[k] - b.sumc2[k]) <= tol, k
    assert abs(a.total_energy - b.total_energy) <= tol


@pytest.mark.parametrize("nroot", [1, 2])
def test_davidson_of_many_chunks(gpu_lib, nroot):
    """43,758 determinants, 43 chunks of 1,024 rows: a lane of the warp that adds the chunks has two.
    Real and complex arithmetic agree, and the energy rebuilt from the density matrices of the
    vector is its root within 1e-10 Eh, as the check of smaller spaces."""
    from dirac_caspt2_gb300 import api
    s = _real((2, 18, 4, 8), 71)
    c = dataclasses.replace(s, realonly=False, rec_val=np.asarray(s.rec_val, np.complex128))
    got = []
    for x in (s, c):
        with api.Caspt2Session(0) as ses:
            ses.set_system(x)
            ses.set_casci_solver("davidson")
            e, n, v = ses.casci(nroot, want_ci=True)
            chk = ses.casci_energy_check()
        assert n == 43758
        v = v[:, :nroot]
        assert np.abs(v.conj().T @ v - np.eye(nroot)).max() <= 1e-12
        assert abs(chk["error"]) <= 1e-10
        got.append(np.asarray(e)[:nroot])
    assert np.abs(got[0] - got[1]).max() <= 1e-11
