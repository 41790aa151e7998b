"""The float32 product on the tensor cores: tiles, tails and cuts of K against float64, the epilogue, and numbers without terms."""
import pytest
import torch

from qstream_b200.csrc import gemm_tc, ops
from qstream_b200.parts.linear import linear

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


# rows and features at the edges of tiles and of a CTA's 128 features, K of one block of 64, with tails, and cut over many pairs of blocks
# (tiles of 256 tokens, and pairs that take several units: below)
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


@pytest.mark.parametrize("K", [256, 4096, 16384])
def test_operands_of_one_sign(K):
    """The unit cuts off where it adds: with operands that are both of one sign, which add up without cancelling, that is a bias.  A run's last four steps
    are what counts: at a quarter, a half, three quarters and all of its sum each cuts off an ulp (2^-23) at most, half of one on average."""
    g = torch.Generator().manual_seed(K)
    for x, w in ((torch.rand(300, K, generator=g), torch.rand(512, K, generator=g)),
                 (torch.relu(torch.randn(300, K, generator=g)) ** 2, torch.rand(512, K, generator=g)),
                 (torch.sigmoid(torch.randn(300, K, generator=g)), torch.randn(512, K, generator=g).abs())):
        x, w = x.cuda(), w.cuda()
        ref = x.double() @ w.double().T
        off = (ops.linear_split(x, w).double() - ref) / ref
        runs = -(-K // 64)
        assert off.abs().max() <= 2.5 * 2.0 ** -23 + (runs + 4) * EPS
        # 2.5 halves of an ulp, an ulp being 0.72 of 2^-23 of a number on average, and the runs' roundings around it
        assert -1.25 * 2.0 ** -23 <= off.mean() <= 0.1 * 2.0 ** -23
        assert off.square().mean().sqrt() <= 1.25 * 2.0 ** -23
    gemm_tc.check_status("cuda:0")


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


@pytest.mark.parametrize("low", [-100, -112, -120, -126])
def test_very_small_operands_are_held_whole(low):
    """Below 2^-109 a number's last bfloat16 term is cut: such sums are taken from the 32-bit numbers, and nobody else's results change."""
    for M, N, K in ((40, 300, 2048), (300, 256, 512), (700, 600, 260)):
        g = torch.Generator().manual_seed(K)
        x, w = torch.randn(M, K, generator=g).cuda(), torch.randn(N, K, generator=g).cuda()
        plain = ops.linear_split(x, w)
        small = x.clone()
        small[M // 2:M // 2 + 3] *= 2.0 ** low
        for a, b in ((small, w), (x, w * 2.0 ** low)):
            got, ref, size = ops.linear_split(a, b), a.double() @ b.double().T, a.double().abs() @ b.double().abs().T
            # runs of 256 products as a chain of rounded additions, then the runs; nothing below 2^-149
            assert ((got.double() - ref).abs() <= (256 + -(-K // 64)) * EPS * size + K * 2.0 ** -149).all()
            if a is small:
                rows = torch.ones(M, dtype=torch.bool)
                rows[M // 2:M // 2 + 3] = False
                assert torch.equal(got[rows], plain[rows])
    gemm_tc.check_status("cuda:0")


@pytest.mark.parametrize("K", [258, 255])
def test_rows_that_are_no_whole_pieces_are_refused(K):
    from qstream_b200 import QStreamError
    x, w = torch.zeros(40, K, device="cuda"), torch.zeros(64, K, device="cuda")
    assert not ops.split_takes(x, w)
    with pytest.raises(QStreamError):
        ops.linear_split(x, w)
    assert linear(x, w).shape == (40, 64)


# (N, K): the forms that their row counts below reach, as (tokens of a tile, whether units of a tile run side by side, whether these hand on runs).
# Tails of rows, features and K; pairs with one unit and with several (over 74), of one tile's parts and of other tiles
FORMS = {(2570, 2564): {(32, True, True), (64, True, True), (128, True, False), (64, True, False), (256, True, False)},
         (6200, 1284): {(32, True, False), (64, True, False), (128, True, False), (256, True, False), (64, False, False), (128, False, False)},
         (4100, 1284): {(32, True, True), (64, True, False), (256, False, False), (256, True, False)},
         (9500, 644): {(32, False, False), (64, False, False), (128, False, False), (256, False, False)},
         (64, 2052): {(32, True, True), (64, True, True)}, (300, 260): {(32, True, True), (64, True, True), (32, False, False)}}
ROWS = (1, 2, 16, 17, 33, 64, 65, 100, 129, 257, 300, 513, 700, 1100)


@pytest.mark.parametrize("N,K", list(FORMS))
def test_a_row_is_the_same_bits_whatever_else_is_in_the_batch(N, K):
    """Every form a product can take, by its number of rows: against float64, and the same bits for each row; among them pairs with several
    units (barriers and stages used on), tiles of 256 tokens, and a number that is not finite in the last unit."""
    forms = {M: ops.linear_split_form(M, N, K) for M in ROWS}
    assert FORMS[N, K] <= {(f[0], f[2] > 1, f[3]) for f in forms.values()}
    assert len({f[1] for f in forms.values()}) == 1
    if N > 2500:
        assert any(-(-M // f[0]) * -(-N // 256) * f[2] > 74 for M, f in forms.items())
    M = max(ROWS)
    g = torch.Generator().manual_seed(N + K)
    x, w, bias = torch.randn(M, K, generator=g).cuda(), (torch.randn(N, K, generator=g) * K ** -0.5).cuda(), torch.randn(N, generator=g).cuda()
    res = (torch.randn(M, N, generator=g).cuda(),)
    whole = linear(x, w, bias, "gelu_new", res)
    ref, size = x.double() @ w.double().T + bias.double(), x.double().abs() @ w.double().abs().T + bias.double().abs()
    ref = torch.nn.functional.gelu(ref, approximate="tanh") + res[0].double()
    # as above for the sum; gelu's slope is below 1.2, its own roundings and those behind it act on values of the size of the sums
    runs = -(-K // 64)
    assert ((whole.double() - ref).abs() <= 1.2 * (2 * 24 + 4 + 2 * runs) * EPS * size + 16 * EPS * (ref.abs() + res[0].abs() + 1)).all()
    for n in ROWS:
        for at in {0, M - n}:
            assert torch.equal(linear(x[at:at + n], w, bias, "gelu_new", (res[0][at:at + n],)), whole[at:at + n]), (n, at, forms[n])
    gemm_tc.check_status("cuda:0")
    x[M - 2, K - 3], x[M - 1, 5] = float("inf"), 3.4e38                 # the second: infinity as a bfloat16 only
    odd = linear(x, w, bias)
    plain = ops.linear_simt(x[M - 2:], w, bias)
    assert torch.equal(torch.isnan(odd[M - 2:]), torch.isnan(plain)) and torch.equal(torch.isinf(odd[M - 2:]), torch.isinf(plain))
    for n in ROWS:
        torch.testing.assert_close(linear(x[M - n:], w, bias), odd[M - n:], rtol=0, atol=0, equal_nan=True)
    gemm_tc.check_status("cuda:0")


def test_the_workspace_that_a_product_takes_is_asked_for():
    from qstream_b200 import QStreamError
    x, w, out = torch.zeros(16, 2048, device="cuda"), torch.zeros(2048, 2048, device="cuda"), torch.zeros(16, 2048, device="cuda")
    lib = ops.library()
    floats = lib.qs_linear_split_scratch(16, 2048, 2048)
    assert floats > 0
    with pytest.raises(QStreamError):
        ops.check(lib.qs_linear_split(ops.ptr(out), ops.ptr(x), ops.ptr(w), None, 0, 0, None, None, 16, 2048, 2048, 2048, 2048, 2048, None, 0,
                                      ops.ptr(gemm_tc.status_word(x.device)), ops.stream()))


def test_a_float32_request_is_the_same_bits_alone_in_a_batch_and_in_portions(tmp_path):
    import qstream_b200 as qs
    cfg = qs.GptjConfig.from_dict(dict(n_layer=2, n_embd=1024, n_head=8, n_positions=256, vocab_size=512, rotary_dim=16,
                                       architectures=["GPTJForCausalLM"]))
    model = qs.load_model(qs.write_model_folder(str(tmp_path / "m"), cfg, seed=3, dtype="float32"), dtype="float32", device="cuda:0")
    g = torch.Generator().manual_seed(1)
    prompts = [torch.randint(0, 512, (n,), generator=g).tolist() for n in (7, 40, 100)]
    engine = qs.Engine(model, max_tokens=1024, max_batch=3)

    def serve(which, portion):
        slots = [engine.acquire() for _ in which]
        rest = [list(prompts[i]) for i in which]
        while any(len(r) > portion for r in rest):          # all but the last portions, a sequence at a time
            for k, r in enumerate(rest):
                if len(r) > portion:
                    engine.step([slots[k]], [r[:portion]])
                    rest[k] = r[portion:]
        out = [engine.step(slots, rest).clone()]
        for t in (5, 17):
            out.append(engine.step(slots, [[t]] * len(which)).clone())
        for s in slots:
            engine.release(s)
        return out

    together = serve((0, 1, 2), 1000)
    for got in (serve((0, 1, 2), 30), serve((0, 1, 2), 9)):
        assert all(torch.equal(a, b) for a, b in zip(together, got))
    for i in range(3):
        for a, b in zip(together, serve((i,), 1000)):
            assert torch.equal(a[i], b[0])
    engine.check_status()
