"""FP64 products with more columns than one launch of small tiles covers (65,535 tiles of 4 columns), in
parts: against torch.matmul in complex128 within 6 (k + 2) u (|A||B|)_ij, u = 2^-53, the bound of the
other FP64 products."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("m,n,k,batch", [(3, 300001, 40, 1), (8, 600002, 40, 1), (5, 270001, 7, 2)])
@pytest.mark.parametrize("conj", [False, True])
def test_many_columns(gpu_lib, m, n, k, batch, conj):
    from dirac_caspt2_gb300 import api
    g = torch.Generator(device="cuda").manual_seed(m + n + k)

    def rnd(*shape):
        return torch.complex(torch.randn(shape, generator=g, device="cuda", dtype=torch.float64),
                             torch.randn(shape, generator=g, device="cuda", dtype=torch.float64))

    A, B = rnd(batch, k, m), rnd(n, k)
    C = torch.zeros((batch, n, m), dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()
    with api.Caspt2Session(0) as ses:
        ses.zgemm(api.DCG_PREC_FP64, m, n, k, batch, A.data_ptr(), 1, m, k * m, B.data_ptr(), k, conj,
                  C.data_ptr(), 1, m, n * m)
    ref = torch.matmul(B.conj() if conj else B, A)
    assert ((C - ref).abs() <= 6 * (k + 2) * 2.0 ** -53 * torch.matmul(B.abs(), A.abs())).all()
