"""Products with few features against float64: tiles of 8, 16, 32 and 64 features and one more, tails of tokens and of K, the epilogue, strides."""
import pytest
import torch

from qstream_b200.csrc import gemm_tc

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


@pytest.mark.parametrize("N", [1, 8, 9, 16, 17, 32, 33, 64, 65])
@pytest.mark.parametrize("M,K", [(1, 8), (15, 4096), (17, 520), (64, 2048), (128, 72), (300, 512), (4096, 64), (4097, 64)])
def test_few_features(M, N, K):
    g = torch.Generator().manual_seed(M + N + K)
    wide, w = torch.randn(M, K + 8, generator=g).bfloat16().cuda(), torch.randn(N, K, generator=g).bfloat16().cuda()
    bias, res = torch.randn(N, generator=g).cuda(), torch.randn(M, N, generator=g).bfloat16().cuda()
    x = wide[:, 8:]
    got = gemm_tc.linear(x, w, bias, None, (res,), torch.float32)
    gemm_tc.check_status("cuda:0")
    ref = x.double() @ w.double().T + bias.double() + res.double()
    size = x.double().abs() @ w.double().abs().T + bias.double().abs() + res.double().abs()
    # an ulp (2 EPS) of what is summed so far per step of 16 products in the unit, and a rounding per run and warp
    assert ((got.double() - ref).abs() <= (2 * (K / 16 + 1) + 40) * EPS * size).all()
    # rows are the same bits in any part of the batch that the same kernel takes, and in a matrix that is part of a wider one
    if N <= 32 and 1 < M <= 4096:
        rows = slice(M // 3, M // 3 + (M + 1) // 2)
        assert torch.equal(gemm_tc.linear(x[rows], w, bias, None, (res[rows],), torch.float32), got[rows])
    view = torch.cat([w, w], 1)[:, :K]
    assert torch.equal(gemm_tc.linear(x, view, bias, None, (res,), torch.float32), got)
    half = gemm_tc.linear(x, w, bias, "gelu")
    assert half.dtype == torch.bfloat16
    ref = torch.nn.functional.gelu(x.double() @ w.double().T + bias.double())
    assert ((half.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1.2 * (2 * (K / 16 + 1) + 40) * EPS * size + 1e-6).all()


@pytest.mark.parametrize("N,K", [(16, 4096), (24, 8192), (33, 2048), (48, 512), (64, 4096)])
def test_a_row_is_the_same_bits_in_any_batch_of_up_to_128(N, K):
    """What the few-token kernels promise their callers holds for few features too."""
    g = torch.Generator().manual_seed(N)
    x, w = torch.randn(128, K, generator=g).bfloat16().cuda(), torch.randn(N, K, generator=g).bfloat16().cuda()
    whole = gemm_tc.linear(x, w, out_dtype=torch.float32)
    for rows in (slice(0, 1), slice(5, 21), slice(0, 63), slice(64, 128), slice(1, 66)):
        assert torch.equal(gemm_tc.linear(x[rows], w, out_dtype=torch.float32), whole[rows])
