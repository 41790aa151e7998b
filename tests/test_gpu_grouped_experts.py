"""Experts whose matrices are read once for all tokens that chose them (few tokens), and all experts' products in one launch (many),
against float64, at the edges of tiles, chunks of tokens and groups."""
import pytest
import torch

from qstream_b200.csrc import gemm_tc, ops

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def i32(t):
    return torch.as_tensor(t, dtype=torch.int32).cuda()


@pytest.mark.parametrize("T,top,E,D,F", [(1, 1, 1, 8, 8), (8, 4, 16, 256, 64), (3, 2, 5, 40, 24), (32, 4, 16, 136, 72), (33, 2, 3, 64, 16), (70, 8, 9, 264, 40),
                                         (20, 1, 1, 72, 104), (9, 16, 40, 48, 56), (31, 3, 70, 512, 16)])
@pytest.mark.parametrize("gated", [False, True])
def test_few_tokens(T, top, E, D, F, gated):
    """Choices among the experts and one output behind them that returns its input; rows of nobody; every token its own sum, the
    same bits alone as in the batch."""
    g = torch.Generator(device="cuda").manual_seed(T * D + F)
    x = torch.randn(T, D + 8, generator=g, device="cuda").to(BF)[:, :D]
    w_up = (torch.randn(E, F * (2 if gated else 1), D, generator=g, device="cuda") * D ** -0.5).to(BF)
    w_down = (torch.randn(E, D, F, generator=g, device="cuda") * F ** -0.5).to(BF)
    n = max(E + 1, top)
    idx = torch.stack([torch.randperm(n, generator=torch.Generator().manual_seed(t))[:top] for t in range(T)]).clamp(max=E).cuda()
    if top <= E and T > 2:
        idx[1] = torch.arange(top)                      # crowds on the first experts
        idx[2] = torch.arange(top)
    wts = torch.rand(T, top, generator=g, device="cuda")
    slots = torch.arange(T, dtype=torch.int32, device="cuda")
    if T > 4:
        slots[3] = -1
    add, scale = torch.randn(T, D, generator=g, device="cuda"), torch.rand(T, generator=g, device="cuda")
    got = ops.moe_experts_indirect(x, w_up, w_down, i32(idx), wts, slots, "silu", add, scale, gated=gated)
    assert got.dtype == torch.float32
    live = slots >= 0
    ref, size = (torch.zeros(T, D, dtype=torch.float64, device="cuda") for _ in range(2))
    ref += torch.where(live[:, None], add.double() * scale.double()[:, None], 0)
    for j in range(top):
        for t in range(T):
            if not live[t]:
                continue
            e = int(idx[t, j])
            if e >= E:
                y, mag = x[t].double(), x[t].double().abs()
            else:
                u = w_up[e].double() @ x[t].double()
                h = torch.nn.functional.silu(u[:F]) * (u[F:] if gated else 1)
                y, mag = w_down[e].double() @ h, w_down[e].double().abs() @ h.abs()
            ref[t] += wts[t, j].double() * y
            size[t] += wts[t, j].double() * mag
    # a hidden element is rounded to a number of eight significant bits: by 2^-8 of it at most; everything else is 32-bit
    assert ((got.double() - ref).abs() <= (2.0 ** -8 + 1e-5) * size + 1e-5).all()
    assert not got[~live].any()
    for t in {0, T - 1, T // 2}:
        one = ops.moe_experts_indirect(x[t:t + 1], w_up, w_down, i32(idx[t:t + 1]), wts[t:t + 1].contiguous(), slots[t:t + 1].contiguous(), "silu",
                                       add[t:t + 1], scale[t:t + 1].contiguous(), gated=gated)
        assert torch.equal(one[0], got[t])


@pytest.mark.parametrize("F", [512, 1024, 4096, 8200])
def test_long_sums_are_rounded_and_not_cut_off(F):
    """The second product alone, on hidden values as they are: positive terms, whose sum loses to a unit that cuts off at every step."""
    T, D = 8, 512
    g = torch.Generator(device="cuda").manual_seed(F)
    hidden, w = ((torch.rand(s, generator=g, device="cuda") + 0.5).to(BF) for s in ((T, F), (1, D, F)))
    x, out = torch.zeros(T, D, dtype=BF, device="cuda"), torch.empty(T, D, device="cuda")
    p, slots = ops.ptr, i32(range(T))
    idx, wts = i32([[0]] * T), torch.ones(T, 1, device="cuda")
    ops.check(ops.library().qs_moe_expert_down(p(out), D, p(hidden), F, p(w), ops.dtype_code(hidden), p(idx), p(wts), p(slots), None, 0, 0, None, T, 1, D, F, p(x), D, 1,
                                               ops.stream()))
    ref = hidden.double() @ w[0].double().T
    off = (out.double() - ref) / ref
    # rounded additions (F / 128 in a row in a quarter of the sum, four behind them) err either way: at most 2^-24 each, nothing on average over
    # the 4,096 results; a product of 16 terms of one size, cut off inside the unit, loses at most 2^-23 and as much again for the terms' sizes
    assert off.abs().max() <= (F / 128 + 4) * 2.0 ** -24 + 2.0 ** -22
    assert off.mean().abs() <= 2.0 ** -22


def took(T, top, E, D, F):
    """Milliseconds of a step of T tokens that choose `top` of E experts each, best of a few, ten steps in a row without the host between them."""
    x, w_up, w_down = torch.randn(T, D, device="cuda").to(BF), torch.zeros(E, 2 * F, D, dtype=BF, device="cuda"), torch.zeros(E, D, F, dtype=BF, device="cuda")
    g = torch.Generator().manual_seed(T)
    idx, wts = i32(torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(T)])), torch.ones(T, top, device="cuda")
    slots, graph, best = i32(range(T)), torch.cuda.CUDAGraph(), []
    step = lambda: ops.moe_experts_indirect(x, w_up, w_down, idx, wts, slots, "silu", gated=True)         # noqa: E731
    step()
    with torch.cuda.graph(graph):
        for _ in range(10):
            step()
    for _ in range(5):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        graph.replay()
        b.record()
        torch.cuda.synchronize()
        best.append(a.elapsed_time(b) / 10)
    return min(best)


def test_many_pairs_cost_no_more_than_their_matrices():
    """The same 64 experts' matrices for four times the pairs, as many as a block takes: putting the pairs in order must not show (it took
    six sevenths of the step when it grew with the square of their number; now the step is a quarter longer)."""
    few, many = took(32, 4, 64, 2048, 512), took(32, 16, 64, 2048, 512)
    assert many <= 2.5 * few, (few, many)


def test_experts_that_nobody_chose_cost_nothing():
    """One token with four of 1,024 experts or of eight: only blocks that have work (with a block per expert it took two to three times as long)."""
    few, many = took(1, 4, 8, 256, 256), took(1, 4, 1024, 256, 256)
    assert many <= 1.5 * few, (few, many)


@pytest.mark.parametrize("counts", [[5], [0, 0, 129, 1, 0, 128, 127], [300, 0, 7], [1] * 70, [40] * 16, [0, 0], [1000, 513]])
@pytest.mark.parametrize("N,K", [(64, 72), (512, 128), (300, 2048), (1024, 512)])
@pytest.mark.parametrize("out_dtype", [torch.float32, BF])
def test_products_of_groups(counts, N, K, out_dtype):
    g = torch.Generator(device="cuda").manual_seed(N + K + len(counts))
    E, tail = len(counts), 9                            # rows behind the last group: left alone
    M = sum(counts) + tail
    x = torch.randn(M, K, generator=g, device="cuda").to(BF)
    x[M - tail:] = float("nan")
    w = (torch.randn(E, N, K, generator=g, device="cuda") * K ** -0.5).to(BF)
    offsets = [0]
    for c in counts:
        offsets.append(offsets[-1] + c)
    out = torch.full((M, N), 7.0, dtype=out_dtype, device="cuda")
    ops.grouped_products(out, x, w, i32(offsets + [M]))
    gemm_tc.check_status("cuda:0")
    for e in range(E):
        sl = slice(offsets[e], offsets[e + 1])
        a, b = x[sl].double(), w[e].double()
        eps = K * 2.0 ** -23 * (a.abs() @ b.abs().T) + (2.0 ** -8 * (a @ b.T).abs() if out_dtype == BF else 0)
        assert ((out[sl].double() - a @ b.T).abs() <= eps).all()
    assert bool((out[M - tail:] == 7.0).all())
