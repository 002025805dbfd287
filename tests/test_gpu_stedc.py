"""The divide-and-conquer tridiagonal eigensolver at the edges of its merge tree (the in-block base
of 32 columns, one more, whole and ragged levels) and on spectra that deflate: by the z test, by
rotations of close poles inside one half and across halves, and in chains.

Bounds: with T = Z diag(w) Z^T computed by a backward-stable method each of |T Z - Z w| and
|Z^T Z - 1| is a small multiple of n u (|T| = its norm, u = 2^-53); 20 n u is allowed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _tridiagonal(kind, n, rng):
    if kind == "random":
        return rng.normal(size=n), rng.normal(size=max(n - 1, 0))
    if kind == "wilkinson":      # pairs of eigenvalues equal to rounding: chains of rotations
        return np.abs(np.arange(n) - (n - 1) / 2.0), np.ones(max(n - 1, 0))
    if kind == "glued":          # blocks with equal spectra joined by tiny couplings
        d = np.abs((np.arange(n) % 21) - 10.0)
        e = np.ones(max(n - 1, 0))
        e[20::21] = 1e-9
        return d, e
    if kind == "pairs":          # every eigenvalue twice, and a null space
        d = np.repeat(np.maximum(rng.normal(size=(n + 1) // 2), 0.0), 2)[:n]
        e = 1e-15 * rng.normal(size=max(n - 1, 0))
        return d, e
    return np.ones(n), np.zeros(max(n - 1, 0))   # "constant"


@pytest.mark.parametrize("n", [1, 2, 3, 17, 31, 32, 33, 63, 64, 65, 97, 130, 257, 700])
@pytest.mark.parametrize("kind", ["random", "wilkinson", "glued", "pairs", "constant"])
def test_stedc_edges(gpu_lib, n, kind):
    from dirac_caspt2_gb300 import api
    d, e = _tridiagonal(kind, n, np.random.default_rng(n))
    with api.Caspt2Session(0) as ses:
        w, Z = ses.stedc(d, e)
    T = np.diag(d) + np.diag(e, 1) + np.diag(e, -1)
    norm = max(np.abs(T).sum(axis=0).max(), 1e-300)
    assert (np.diff(w) >= 0).all()
    assert np.abs(w - np.linalg.eigvalsh(T)).max() <= 20 * n * U * norm
    assert np.abs(T @ Z - Z * w).max() <= 20 * n * U * norm
    assert np.abs(Z.T @ Z - np.eye(n)).max() <= 20 * n * U


@pytest.mark.parametrize("n,vlo", [(20, 0), (33, 5), (64, 63), (200, 150), (300, 1)])
def test_vectors_of_a_range(gpu_lib, n, vlo):
    """Only the last merge's wanted columns are formed."""
    from dirac_caspt2_gb300 import api
    rng = np.random.default_rng(n)
    G = rng.normal(size=(n, n // 2 + 1)) + 1j * rng.normal(size=(n, n // 2 + 1))
    A = G @ G.conj().T           # half the spectrum zero
    with api.Caspt2Session(0) as ses:
        w, Z = ses.heev_range(A, vlo)
        w2, Z2 = ses.heev_range(A, 0)
    norm = np.linalg.norm(A, 2)
    assert np.array_equal(w, w2)
    for v, z in ((vlo, Z), (0, Z2)):
        assert np.abs(A @ z - z * w[v:]).max() <= 20 * n * U * norm
        assert np.abs(z.conj().T @ z - np.eye(n - v)).max() <= 20 * n * U
