"""The rotation by halves and the cache write in 16-byte pieces against float64, and where rows do not allow pieces."""
import pytest
import torch

from qstream_b200.csrc import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dh,dv,R", [(16, 16, 16), (64, 64, 32), (128, 128, 64), (128, 64, 128), (96, 104, 48), (72, 72, 8), (64, 64, 24)])
@pytest.mark.parametrize("T,shift", [(5, 0), (300, 0), (40, 1)])
@pytest.mark.parametrize("first", [False, True])
def test_rotation_by_halves_in_pieces(dh, dv, R, T, shift, first):
    """`shift`: rows that begin off a 16-byte boundary, which the general kernel takes; R / 2 = 4 and 12 go there too."""
    H, G = 4, 2
    g = torch.Generator().manual_seed(dh + R + T)
    row = torch.randn(T, H * dh + G * (dh + dv) + 8, generator=g).bfloat16().cuda()
    at = [shift, shift + H * dh, shift + (H + G) * dh, shift + (H + G) * dh + G * dv]
    q, k, v = (row[:, a:b] for a, b in zip(at, at[1:]))
    vf = torch.randn(T, G * dv, generator=g).bfloat16().cuda() if first else None
    q0, k0, v0 = (x.clone() for x in (q, k, v))
    ang = torch.rand(T, R // 2, generator=g, dtype=torch.float64) * 6
    table = torch.stack([torch.cos(ang), torch.sin(ang)], 2).reshape(T, R).float().cuda()
    pages = -(-T // 64)
    order = torch.randperm(pages + 2, generator=g)[:pages].int()
    kc, vc = torch.full((pages + 2, G, 64, dh), 7.0).bfloat16().cuda(), torch.full((pages + 2, G, 64, dv), 7.0).bfloat16().cuda()
    slot, pos = torch.zeros(T, dtype=torch.int32), torch.arange(T, dtype=torch.int32)
    slot[1] = -1
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    ops.rope_store(q, k, v, H, G, dh, R, table, slot.cuda(), pos.cuda(), order[None].cuda(), 64, kc, vc, status, v_head_dim=dv, v_first=vf, v_mix=0.25,
                   half_layout=True)
    assert int(status.item()) == 0

    def turned(x, n):
        x = x.double().view(T, n, dh).clone()
        c, s = table[:, None, 0::2].double(), table[:, None, 1::2].double()
        a, b = x[..., :R // 2].clone(), x[..., R // 2:R].clone()
        x[..., :R // 2], x[..., R // 2:R] = a * c - b * s, a * s + b * c
        return x

    live = slot >= 0
    near = lambda got, ref: bool(((got.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5).all())        # noqa: E731
    assert near(q.view(T, H, dh)[live], turned(q0, H)[live]) and torch.equal(q[~live], q0[~live])
    where = order.long()[pos.long() // 64].cuda(), pos.long().cuda() % 64
    assert near(kc[where[0], :, where[1]][live], turned(k0, G)[live])
    value = v0.double().view(T, G, dv) if vf is None else 0.75 * v0.double().view(T, G, dv) + 0.25 * vf.double().view(T, G, dv)
    assert near(vc[where[0], :, where[1]][live], value[live])
    assert bool((kc[where[0], :, where[1]][~live] == 7.0).all()) and torch.equal(k, k0) and torch.equal(v, v0)
