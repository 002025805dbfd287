"""The FP64 complex GEMM (dcg_zgemm, DCG_PREC_FP64) at the edges of its tiles, chunks of K and K
splits against torch.matmul in complex128.

Bound per element: a real part is a sum of 2k products, so its rounding error is at most 2 k u
sum |a||b| (u = 2^-53), the complex element's sqrt(2) times that, and the reference's the same:
6 (k + 2) u (|A||B|)_ij."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("m,n,k,batch", [
    (1, 1, 1, 1), (7, 3, 5, 1), (8, 4, 32, 1), (9, 5, 33, 3), (16, 16, 16, 1), (17, 13, 47, 2), (33, 31, 100, 1),
    (14, 14, 2744, 1), (1, 288, 924, 1), (65, 63, 129, 1), (66, 1000, 66, 1), (300, 7, 1000, 1), (130, 200, 64, 5),
    (792, 20, 792, 1), (200, 3, 12, 40)])
@pytest.mark.parametrize("conj,accumulate", [(False, False), (True, True)])
def test_fp64_gemm_edges(gpu_lib, m, n, k, batch, conj, accumulate):
    from dirac_caspt2_gb300 import api
    g = torch.Generator(device="cuda").manual_seed(m + 3 * n + 7 * k + batch)
    def rnd(*shape):
        return torch.complex(torch.randn(shape, generator=g, device="cuda", dtype=torch.float64),
                             torch.randn(shape, generator=g, device="cuda", dtype=torch.float64))
    pad = 3                                                 # leading dimensions beyond the matrices
    A, B, C = rnd(batch, k, m + pad), rnd(n, k + pad), rnd(batch, n, m + pad)
    C0 = C.clone()
    torch.cuda.synchronize()
    with api.Caspt2Session(0) as ses:
        ses.zgemm(api.DCG_PREC_FP64, m, n, k, batch, A.data_ptr(), 1, m + pad, k * (m + pad), B.data_ptr(), k + pad, conj,
                  C.data_ptr(), 1, m + pad, n * (m + pad), accumulate=accumulate)
    Am, Bm = A[:, :, :m], B[:, :k]
    ref = torch.matmul(Bm.conj() if conj else Bm, Am)
    if accumulate:
        ref = ref + C0[:, :, :m]
    bound = 6 * (k + 2) * 2.0 ** -53 * (torch.matmul(Bm.abs(), Am.abs()) + (C0[:, :, :m].abs() if accumulate else 0))
    assert ((C[:, :, :m] - ref).abs() <= bound).all()
    assert torch.equal(C[:, :, m:], C0[:, :, m:])           # nothing written beyond the rows
