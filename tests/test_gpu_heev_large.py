"""Hermitian eigendecomposition around the order where the reduction leaves shared memory for
columns in global memory (about 1,290 on 152 SMs) and above, complex and real: residuals and
orthogonality within 20 n u (a backward-stable method's few n u, u = 2^-53), on a rank-deficient
Gram matrix, and the given-up wait of that kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
U = 2.0 ** -53


def _gram(n, real):
    g = torch.Generator(device="cuda").manual_seed(n)
    X = torch.randn(n, (2 * n) // 3, generator=g, device="cuda", dtype=torch.float64)
    if not real:
        X = torch.complex(X, torch.randn(X.shape, generator=g, device="cuda", dtype=torch.float64))
    return X @ X.conj().T


@pytest.mark.parametrize("n", [1280, 1300, 1409, 1793])
@pytest.mark.parametrize("real", [False, True])
def test_decomposition(gpu_lib, n, real):
    from dirac_caspt2_gb300 import api
    A = _gram(n, real)
    with api.Caspt2Session(0) as ses:
        w, z = ses.heev(A.cpu().numpy())
    assert (np.diff(w) >= 0).all()
    Z, W = torch.from_numpy(z).cuda(), torch.from_numpy(w).cuda()
    A = A.to(Z.dtype)
    assert float((A @ Z - Z * W).abs().max()) <= 20 * n * U * float(W.abs().max())
    assert float((Z.conj().T @ Z - torch.eye(n, device="cuda")).abs().max()) <= 20 * n * U


def test_wait_runs_out_and_context_recovers(gpu_lib):
    from dirac_caspt2_gb300 import api
    A = _gram(1500, False).cpu().numpy()
    with api.Caspt2Session(0) as ses:
        ref = ses.heev(A, vectors=False)
        ses.set_wait_limit(1e-9)
        raised = 0
        for _ in range(3):
            try:
                assert np.array_equal(ses.heev(A, vectors=False), ref)   # no wait ran out
            except api.DcgError as e:
                assert e.code == -6 and "timed out" in str(e)
                raised += 1
        assert raised > 0
        ses.set_wait_limit(0)
        assert np.array_equal(ses.heev(A, vectors=False), ref)
