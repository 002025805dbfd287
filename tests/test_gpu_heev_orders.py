"""Hermitian eigendecomposition beyond the columns-in-global-memory reduction (about 4,750 rows): the
persistent kernel with grid barriers up to 7,000 rows, one set of launches per column above.  The
matrix is a known real spectrum under two complex reflections, dense, so that the eigenvalues need
no host solver; the top vectors by their residuals.  20 n u each, u = 2^-53."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _known(n):
    """Eigenvalues (ascending) and (1 - 2 v v^H)(1 - 2 u u^H) D (1 - 2 u u^H)(1 - 2 v v^H)."""
    rng = np.random.default_rng(n)
    d = np.sort(rng.normal(size=n))
    A = np.diag(d).astype(complex)
    for _ in range(2):
        u = rng.normal(size=n) + 1j * rng.normal(size=n)
        u /= np.linalg.norm(u)
        p = A @ u
        q = 2.0 * (p - np.vdot(u, p).real * u)
        A -= np.outer(q, u.conj()) + np.outer(u, q.conj())
    i = np.arange(n)
    A[i, i] = A[i, i].real
    return d, A


@pytest.mark.parametrize("n", [4900, 7001])
def test_known_spectrum(gpu_lib, n):
    from dirac_caspt2_gb300 import api
    d, A = _known(n)
    with api.Caspt2Session(0) as ses:
        w, Z = ses.heev_range(A, n - 3)
    norm = np.abs(d).max()
    assert np.abs(w - d).max() <= 20 * n * U * norm
    assert np.abs(A @ Z - Z * w[n - 3:]).max() <= 20 * n * U * norm
    assert np.abs(Z.conj().T @ Z - np.eye(3)).max() <= 20 * n * U


def test_grid_barrier_runs_out_and_context_recovers(gpu_lib):
    from dirac_caspt2_gb300 import api
    d, A = _known(4900)
    with api.Caspt2Session(0) as ses:
        ses.set_wait_limit(1e-9)
        raised = 0
        for _ in range(3):   # a wait gives up once a block has polled for longer than the limit
            try:
                assert np.abs(ses.heev(A, vectors=False) - d).max() <= 20 * 4900 * U * np.abs(d).max()
            except api.DcgError as e:
                assert e.code == -6 and "timed out" in str(e)
                raised += 1
        assert raised > 0
        ses.set_wait_limit(0)
        assert np.abs(ses.heev(A, vectors=False) - d).max() <= 20 * 4900 * U * np.abs(d).max()
