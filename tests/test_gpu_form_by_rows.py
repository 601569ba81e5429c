"""The narrow GEMM tiles whose Q4_K min term has its own accumulator."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,n,k", [(17, 12800, 256), (32, 12800, 2304), (33, 12800, 768), (49, 256, 4096), (64, 1024, 1024), (65, 1024, 1024)])
def test_min_term_of_narrow_tiles(torch_cuda, rows, n, k):
    """Q4_K products with the min term in its own accumulator (tiles of up to 64 positions) and joined (65 rows), rows of zeros and
    of one value included (d = 0, a min term alone), against 64-bit arithmetic on the same int8 rows.  A sum of K / 256 block
    terms, each rounded a few times, of values that cancel to about a third: 4 sqrt(K / 256) 2^-24."""
    torch = torch_cuda
    from candle_b200 import GgmlDType, QMatMul, QTensor, _lib
    g = torch.Generator(device="cuda").manual_seed(n + k)
    w = torch.randn((n, k), generator=g, device="cuda") * 0.02
    w[3] = 0.0
    w[5] = -0.01
    w[6, :256] = -0.01
    q = QTensor.quantize(w, GgmlDType.Q4K)
    x = torch.randn((rows, k), generator=g, device="cuda")
    qs, sc = torch.empty((rows, k), dtype=torch.int8, device="cuda"), torch.empty((rows, k // 256), device="cuda")
    bs = torch.empty((rows, k // 16), dtype=torch.int16, device="cuda")
    assert _lib.load().candle_moe_quantize_act(torch.cuda.current_stream().cuda_stream, x.data_ptr(), rows, k, 12, qs.data_ptr(), sc.data_ptr(),
                                               bs.data_ptr()) == 0
    a = (qs.double().view(rows, -1, 256) * sc.double()[:, :, None]).view(rows, k)
    ref = a @ q.dequantize().double().to("cuda").T
    got = QMatMul(q).forward(x).double()
    assert torch.isfinite(got).all()
    assert float((got - ref).norm() / ref.norm()) < 4 * (k / 256) ** 0.5 * 2 ** -24
    for r in (3, 5, 6):
        assert float((got[:, r] - ref[:, r]).abs().max()) <= 1e-5 * max(1.0, float(ref[:, r].abs().max()))
