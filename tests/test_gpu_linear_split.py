"""The float32 product on the tensor cores: tiles, tails and cuts of K against float64, the epilogue, and numbers without terms."""
import pytest
import torch

from qstream_b200.csrc import gemm_tc, ops
from qstream_b200.parts.linear import linear

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


# rows at the edges of the four tiles (32, 64, 128, 256 tokens) and of several, features at the edge of 256 and of a CTA's 128, K of one
# block of 64, with tails, and cut over many pairs of blocks
@pytest.mark.parametrize("M,N,K", [(1, 1, 4), (17, 16, 256), (32, 256, 64), (33, 257, 68), (64, 300, 260), (65, 129, 2048), (128, 2048, 1024), (129, 128, 516),
                                   (255, 520, 320), (257, 2048, 2048), (700, 1000, 512), (300, 64, 8192)])
def test_product_against_float64(M, N, K):
    g = torch.Generator().manual_seed(M + N + K)
    x, w = torch.randn(M, K, generator=g).cuda(), torch.randn(N, K, generator=g).cuda()
    got = ops.linear_split(x, w)
    gemm_tc.check_status("cuda:0")
    ref, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    # a run of 64 products: the unit cuts off the sums of 24 steps, in the worst case an ulp (2 EPS) of what is summed each, the terms that are left
    # out are below 4 EPS; then one rounding per run, and per part of K
    runs = -(-K // 64)
    assert ((got.double() - ref).abs() <= (2 * 24 + 4 + 2 * runs) * EPS * size).all()
    # as a whole no further from 64 bits than the CUDA-core product
    far = lambda y: float((y.double() - ref).norm())      # noqa: E731
    assert far(got) <= far(ops.linear_simt(x, w)) * 1.05 + EPS * float(ref.norm())
    assert torch.equal(got, ops.linear_split(x, w))


def test_rows_apart_and_epilogue():
    g = torch.Generator().manual_seed(3)
    for M, N, K in ((40, 300, 2048), (200, 512, 260)):
        wide = torch.randn(M, K + 8, generator=g).cuda()
        w, bias = torch.randn(N, K, generator=g).cuda() * K ** -0.5, torch.randn(N, generator=g).cuda()
        res = [torch.randn(M, N, generator=g).cuda() for _ in range(2)]
        for at in (0, 3, 4):                            # 16-byte aligned rows, which the tensor cores take, and others
            x = wide[:, at:at + K]
            assert ops.split_takes(x, w) == (at != 3)
            for act, f in (("silu", lambda u: u * torch.sigmoid(u)), ("gelu_new", lambda u: torch.nn.functional.gelu(u, approximate="tanh")), (None, lambda u: u)):
                out = torch.full((M, N + 5), 7.0, device="cuda")
                linear(x, w, bias, act, tuple(res), out=out[:, 2:2 + N])
                ref = f(x.double() @ w.double().T + bias.double()) + res[0].double() + res[1].double()
                # slopes below 1.2; the products' bound (either kernel's) and a handful of roundings of values around one
                bound = 1.2 * (256 + -(-K // 64)) * EPS * (x.double().abs() @ w.double().abs().T + 1) + 16 * EPS * (ref.abs() + 1)
                assert ((out[:, 2:2 + N].double() - ref).abs() <= bound).all()
                assert bool((out[:, :2] == 7.0).all()) and bool((out[:, 2 + N:] == 7.0).all())
    gemm_tc.check_status("cuda:0")


def test_numbers_without_terms_give_what_a_plain_product_gives():
    """Infinities, NaN and numbers that round to infinity as bfloat16, in both operands, with K in one part and in several."""
    for M, N, K in ((100, 600, 512), (300, 256, 4096)):
        g = torch.Generator().manual_seed(K)
        x, w = torch.randn(M, K, generator=g).cuda(), (torch.randn(N, K, generator=g) * 0.01).cuda()
        plain = ops.linear_split(x, w)
        x[3, 7], x[50, 100], x[60, 5], w[201, 9] = float("inf"), 3.4e38, float("nan"), -float("inf")
        got, ref = ops.linear_split(x, w), ops.linear_simt(x, w)
        gemm_tc.check_status("cuda:0")
        assert torch.equal(torch.isnan(got), torch.isnan(ref)) and torch.equal(torch.isinf(got), torch.isinf(ref))
        big = torch.isfinite(ref[50])
        torch.testing.assert_close(got[50][big], ref[50][big], rtol=256 * EPS, atol=0)
        rows, cols = torch.ones(M, dtype=torch.bool), torch.ones(N, dtype=torch.bool)
        rows[[3, 50, 60]], cols[201] = False, False
        assert torch.equal(got[rows][:, cols], plain[rows][:, cols])      # nobody else's results change


@pytest.mark.parametrize("K", [258, 255])
def test_rows_that_are_no_whole_pieces_are_refused(K):
    from qstream_b200 import QStreamError
    x, w = torch.zeros(40, K, device="cuda"), torch.zeros(64, K, device="cuda")
    assert not ops.split_takes(x, w)
    with pytest.raises(QStreamError):
        ops.linear_split(x, w)
    assert linear(x, w).shape == (40, 64)
