"""The kernels around a prompt's routed experts: the gated unit inside the grouped product, the choice, the order by expert."""
import numpy as np
import pytest
import torch

from qstream_b200.csrc import gemm_tc, ops

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


# groups at the edges of a tile's 128 rows, empty ones, columns at the edges of half a tile (64 and 128), both tile widths
@pytest.mark.parametrize("counts,F,K", [([1, 0, 127, 128, 129], 64, 72), ([300, 5, 0, 700], 200, 136), ([0, 0, 3], 65, 8), ([1000] * 16, 512, 256), ([33] * 40, 129, 64)])
def test_gated_unit_in_the_grouped_product(counts, F, K):
    g = torch.Generator().manual_seed(F + K)
    E, M = len(counts), sum(counts)
    x = torch.randn(M, K, generator=g).to(BF).cuda()
    w = (torch.randn(E, 2 * F, K, generator=g) * K ** -0.5).to(BF).cuda()
    offsets = torch.tensor(np.concatenate([[0], np.cumsum(counts)]), dtype=torch.int32).cuda()
    out = torch.full((M + 1, F), 7.0, dtype=BF, device="cuda")
    ops.grouped_products(out[:M], x, w, offsets, glu=True)
    wide = torch.empty((M, F), device="cuda")
    ops.grouped_products(wide, x, w, offsets, glu=True)
    gemm_tc.check_status("cuda:0")
    at = 0
    for e, n in enumerate(counts):
        u = x[at:at + n].double() @ w[e].double().T
        ref = torch.nn.functional.silu(u[:, :F]) * u[:, F:]
        # sums of K products in the unit (an ulp of what is summed per 16), through silu's slope of at most 1.1 and the other factor
        size = x[at:at + n].double().abs() @ w[e].double().abs().T
        err = 2.0 ** -23 * (K / 16 + 4) * (1.1 * size[:, :F] * u[:, F:].abs() + u[:, :F].abs() * size[:, F:]) + 1e-6 * ref.abs() + 1e-6
        assert ((wide[at:at + n].double() - ref).abs() <= err).all()
        assert ((out[at:at + n].double() - ref).abs() <= err + 2.0 ** -8 * ref.abs()).all()
        at += n
    assert bool((out[M] == 7.0).all())


@pytest.mark.parametrize("T,E,top,nan", [(5, 16, 4, None), (33, 3, 3, None), (9, 40, 8, 0), (9, 40, 8, 7), (2, 1024, 16, None), (7, 1, 1, None)])
def test_choice(T, E, top, nan):
    """Equal scores go to the lower index; NaN is chosen where a walk in order chooses it: as the first live expert."""
    g = torch.Generator().manual_seed(T * E)
    z = torch.randint(-4, 5, (T, E), generator=g).float()                 # many equal scores
    if nan is not None:
        z[1, nan] = float("nan")
    idx, wts, _ = ops.moe_route(z.cuda(), None, E, top, 1, 1, 1.0)
    s = torch.sigmoid(z.cuda()).cpu().numpy()
    for t in range(T):
        live = s[t].copy()
        for j in range(top):
            best = -1
            for e in range(E):
                if live[e] != -np.inf and (best < 0 or live[e] > live[best]):
                    best = e
            assert int(idx[t, j]) == best
            np.testing.assert_allclose(float(wts[t, j]), s[t, best], rtol=1e-6)
            live[best] = -np.inf


@pytest.mark.parametrize("T,top,E", [(1, 1, 1), (40, 4, 16), (1000, 8, 9), (3000, 4, 16), (77, 16, 300)])
def test_order_by_expert(T, top, E):
    g = torch.Generator().manual_seed(T)
    idx = torch.stack([torch.randperm(max(E, top), generator=g)[:top] for _ in range(T)]).clamp(max=E - 1).int().cuda()
    offsets, place_token, pair_place = ops.moe_sort(idx, E)
    counts = torch.bincount(idx.flatten().long().cpu(), minlength=E)
    assert offsets.cpu().tolist()[:E + 1] == [0, *torch.cumsum(counts, 0).tolist()]
    place = pair_place.flatten().long().cpu()
    assert sorted(place.tolist()) == list(range(T * top))
    assert torch.equal(place_token.cpu()[place], torch.arange(T).repeat_interleave(top).int())
    owner = torch.searchsorted(offsets.cpu()[1:E + 1].contiguous(), place.int(), right=True)
    assert torch.equal(owner, idx.flatten().long().cpu())
