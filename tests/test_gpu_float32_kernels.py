"""The float32 engine's product and prompt attention: every form a size can take, against float64 and against each other."""
import numpy as np
import pytest
import torch

from qstream_b200.csrc import ops
from test_gpu_kernels import PagedCase

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


# sizes at the edges of the three tiles (128 x 128, 64 x 64, 16 x 128), of a run of 256 products and of a cut of K: from
# few rows to many, K within a run, a run exactly, several, and not a multiple of four
@pytest.mark.parametrize("M,N,K", [(1, 200, 2048), (16, 129, 4096), (17, 128, 1025), (70, 2048, 2048), (130, 260, 256), (300, 64, 515),
                                   (700, 2048, 512), (129, 4100, 258), (640, 1280, 8192)])
def test_product_forms(M, N, K):
    g = torch.Generator().manual_seed(M + N + K)
    x, w = torch.randn(M, K, generator=g), torch.randn(N, K, generator=g)
    got = ops.linear_simt(x.cuda(), w.cuda())
    ref, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    # two levels of sums: at most 256 + ceil(K / 256) roundings act on any product
    bound = (256 + -(-K // 256)) * EPS * size
    assert ((got.cpu().double() - ref).abs() <= bound).all()
    # a row is the same bits in every form that its number of rows picks
    for rows in ([0], list(range(min(M, 5))), list(range(M // 2, M))):
        assert torch.equal(ops.linear_simt(x[rows].cuda(), w.cuda()), got[rows])


def test_product_rows_apart_and_epilogue():
    """Rows with a stride, a view as the output, bias, activation and two residuals, where K is cut and where it is not."""
    g = torch.Generator().manual_seed(3)
    for M, N, K in ((9, 300, 2048), (200, 512, 300)):
        wide = torch.randn(M, K + 8, generator=g).cuda()
        w, bias = torch.randn(N, K, generator=g).cuda() * K ** -0.5, torch.randn(N, generator=g).cuda()
        res = [torch.randn(M, N, generator=g).cuda() for _ in range(2)]
        for at in (0, 3, 4):                            # 16-byte aligned rows and others
            x = wide[:, at:at + K]
            out = torch.full((M, N + 5), 7.0, device="cuda")
            ops.linear_simt(x, w, bias, "silu", tuple(res), out=out[:, 2:2 + N])
            u = x.double() @ w.double().T + bias.double()
            ref = u * torch.sigmoid(u) + res[0].double() + res[1].double()
            # silu's slope is below 1.1; the epilogue adds a handful of roundings of values around one
            bound = 1.1 * (256 + -(-K // 256)) * EPS * (x.double().abs() @ w.double().abs().T + 1) + 16 * EPS * (ref.abs() + 1)
            assert ((out[:, 2:2 + N].double() - ref).abs() <= bound).all()
            assert bool((out[:, :2] == 7.0).all()) and bool((out[:, 2 + N:] == 7.0).all())


def attention_args(dh, dv, H, G, maps, lens, seed, page_tokens=64):
    case = PagedCase("float32", lens, 1, G, maps * dh, page_tokens=page_tokens, seed=seed, fill=0.0)
    g = torch.Generator().manual_seed(seed + 1)
    n_pages = case.k_cache.shape[0]
    case.k_cache.copy_(torch.randn(n_pages, G, page_tokens, maps * dh, generator=g))
    case.v_cache = torch.randn(n_pages, G, page_tokens, dv, generator=g).cuda()
    slot = torch.tensor([s for s, n in zip(case.slots, lens) for _ in range(n)], dtype=torch.int32)
    pos = torch.tensor([p for n in lens for p in range(n)], dtype=torch.int32)
    q = torch.randn(sum(lens), H * dh, generator=g).cuda()
    return case, q, slot, pos


@pytest.mark.parametrize("dh,dv,H,G,maps", [(64, 64, 4, 2, 1), (128, 128, 2, 2, 1), (256, 256, 2, 1, 1), (36, 100, 4, 1, 1), (32, 64, 8, 2, 2), (4, 4, 1, 1, 1)])
@pytest.mark.parametrize("mask", [{}, {"window": 37}, {"window": 70, "keep_first": 5}, {"chunk": 50}, {"window": 16, "keep_first": 70}])
def test_tiles_of_queries_are_the_same_bits(dh, dv, H, G, maps, mask):
    """Prompts of several sequences (tiles that span them, padding rows, pages of other sizes): the kernel over 64 queries
    gives the bits of the kernel with a warp per query, which the plain model is compared with elsewhere."""
    lens = [1, 130, 64, 77]
    for page_tokens in (64, 16):
        case, q, slot, pos = attention_args(dh, dv, H, G, maps, lens, dh + dv + page_tokens, page_tokens)
        slot[20], slot[133] = -1, -1                    # padding inside a sequence's rows
        sink = torch.randn(H, generator=torch.Generator().manual_seed(9)).cuda()
        for softcap, sk in ((0.0, None), (20.0, sink)):
            args = (q, H, G, dh, dh ** -0.5, mask.get("window", 0), slot.cuda(), pos.cuda(), case.table.cuda(), page_tokens, case.k_cache,
                    case.v_cache, case.status)
            kw = dict(v_head_dim=dv, softcap=softcap, chunk=mask.get("chunk", 0), keep_first=mask.get("keep_first", 0), sink=sk, maps=maps)
            by_row = ops.attention(*args, **kw)
            tiled = ops.attention(*args, **kw, n_seq=len(lens))
            assert int(case.status.item()) == 0
            assert torch.equal(by_row, tiled)
            assert bool(torch.isfinite(tiled).all()) and not bool(tiled[20].any()) and not bool(tiled[133].any())


def mixed_step(lens, before, H, dh, seed):
    """A step in which sequence i brings lens[i] tokens behind before[i] cached ones, with three rows of nobody behind."""
    case = PagedCase("float32", [a + b for a, b in zip(lens, before)], 1, H, dh, seed=seed, n_slots=len(lens), fill=0.0)
    g = torch.Generator().manual_seed(seed)
    case.k_cache.copy_(torch.randn(case.k_cache.shape, generator=g))
    case.v_cache.copy_(torch.randn(case.v_cache.shape, generator=g))
    slot = torch.tensor([s for s, n in zip(case.slots, lens) for _ in range(n)] + [-1] * 3, dtype=torch.int32).cuda()
    pos = torch.tensor([b + i for n, b in zip(lens, before) for i in range(n)] + [0] * 3, dtype=torch.int32).cuda()
    start = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32).cuda()
    q = torch.randn(sum(lens) + 3, H * dh, generator=g).cuda()
    assert slot.numel() == pos.numel() == q.shape[0]
    args = (q, H, H, dh, dh ** -0.5, 0, slot, pos, case.table.cuda(), 64, case.k_cache, case.v_cache, case.status)
    return case, args, dict(n_seq=len(lens), seq_start=start, longest=max(a + b for a, b in zip(lens, before)))


@pytest.mark.parametrize("lens,before", [([130], [0]), ([64, 64], [0, 0]), ([1] * 40 + [900], [77] * 40 + [0]), ([16, 17, 63, 64, 65, 129], [200, 0, 3, 64, 1, 0]),
                                         ([700, 1, 1], [0, 300, 64]), ([33] * 35, [5 * i for i in range(35)])])
def test_tiles_within_a_sequence_are_the_same_bits(lens, before):
    """Tiles that begin where a sequence begins, one to more sequences than a warp looks at together, among them single rows."""
    case, args, hints = mixed_step(lens, before, 2, 64, len(lens) + lens[0])
    by_row, tiled = ops.attention(*args), ops.attention(*args, **hints)
    assert int(case.status.item()) == 0 and torch.equal(by_row, tiled) and not bool(tiled[sum(lens):].any())


def test_a_prompt_among_decoding_sequences_takes_no_longer_in_tiles():
    """A long prompt beside 64 sequences that bring one token each: their walks run side by side (one after the other in the blocks
    that hold them, the step took 1.7 times as long as with a warp per query; side by side about a quarter)."""
    _, args, hints = mixed_step([1200] + [1] * 64, [0] + [1500] * 64, 4, 128, 3)
    took = {}
    for name, kw in (("tiles", hints), ("rows", {})):
        times = []
        for _ in range(4):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            ops.attention(*args, **kw)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        took[name] = min(times)
    assert took["tiles"] <= took["rows"], took


def test_tiles_keep_what_is_not_finite_to_the_rows_that_see_it():
    lens = [150]
    case, q, slot, pos = attention_args(64, 64, 2, 2, 1, lens, 5)
    page = int(case.table[case.slots[0], 1])
    case.v_cache[page, 1, 30, 7] = float("inf")         # position 94, head 1
    case.k_cache[page, 0, 40] = float("nan")            # position 104, head 0
    args = (q, 2, 2, 64, 0.125, 0, slot.cuda(), pos.cuda(), case.table.cuda(), 64, case.k_cache, case.v_cache, case.status)
    tiled, by_row = ops.attention(*args, n_seq=1), ops.attention(*args)
    assert bool(torch.isfinite(tiled[:94]).all()) and bool(torch.isfinite(tiled[:104, :64]).all())
    np.testing.assert_array_equal(tiled.cpu().numpy(), by_row.cpu().numpy())


def test_a_page_that_is_not_held_is_reported():
    case, q, slot, pos = attention_args(64, 64, 2, 2, 1, [150], 6)
    case.table[case.slots[0], 1] = -1
    args = (q, 2, 2, 64, 0.125, 0, slot.cuda(), pos.cuda(), case.table.cuda(), 64, case.k_cache, case.v_cache, case.status)
    tiled = ops.attention(*args, n_seq=1)
    assert int(case.status.item()) == 3
    case.status.zero_()
    assert torch.equal(tiled, ops.attention(*args)) and int(case.status.item()) == 3
