"""Eigenvectors of reducible matrices: at a block's end a Householder reflector is the identity and is
skipped, alone or a few in a row, in the kernels that share a column between two warps (more
than 256 rows).  Residual and orthogonality within 20 n u (a backward-stable method's few n u,
u = 2^-53), and the same bits on a second run."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _blocks(n, real, rng):
    A = np.zeros((n, n), complex)
    at = 0
    while at < n:
        b = min(int(rng.choice([1, 2, 3, 5, 17, 40])), n - at)
        X = rng.normal(size=(b, b)) + (0 if real else 1j) * rng.normal(size=(b, b))
        A[at:at + b, at:at + b] = X + X.conj().T
        at += b
    return A


@pytest.mark.parametrize("n", [260, 300, 600, 850, 1000])
@pytest.mark.parametrize("real", [False, True])
@pytest.mark.parametrize("nvec", [None, 6])   # all vectors; a few (the prefetching form)
def test_decomposition_of_blocks(gpu_lib, n, real, nvec):
    from dirac_caspt2_gb300 import api
    A = _blocks(n, real, np.random.default_rng(n))
    v0 = 0 if nvec is None else n - nvec
    with api.Caspt2Session(0) as ses:
        w, Z = ses.heev_range(A, v0)
        w2, Z2 = ses.heev_range(A, v0)
    assert np.array_equal(w, w2) and np.array_equal(Z, Z2)
    norm = np.abs(w).max()
    assert np.abs(w - np.linalg.eigvalsh(A)).max() <= 20 * n * U * norm
    assert np.abs(A @ Z - Z * w[v0:]).max() <= 20 * n * U * norm
    assert np.abs(Z.conj().T @ Z - np.eye(n - v0)).max() <= 20 * n * U
