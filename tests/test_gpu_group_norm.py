"""The gated norms in groups, in 16-byte pieces and element by element: sizes and strides at the edges of the choice."""
import pytest
import torch

from qstream_b200.csrc import ops

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16
ACT = {"sigmoid": torch.sigmoid, "silu": torch.nn.functional.silu}


def close(got, ref, terms):
    """32-bit sums of `terms` squares, a root, a quotient and the functions, each a few roundings; then one rounding to the type."""
    eps = 2.0 ** -24 * (terms + 32) + (2.0 ** -8 if got.dtype == torch.bfloat16 else 0)
    assert ((got.double() - ref).abs() <= eps * ref.abs() + 1e-30).all()


@pytest.mark.parametrize("n,group", [(2048, 2048), (2048, 128), (2048, 64), (8192, 8192), (4096, 256), (8200, 8200), (96, 8), (40, 40), (24, 12), (96, 0), (4104, 4104), (2056, 2056)])
@pytest.mark.parametrize("types", [(torch.float32, torch.bfloat16, torch.bfloat16), (torch.float32, torch.float32, torch.float32),
                                   (torch.float32, torch.float32, torch.bfloat16), (torch.bfloat16, torch.bfloat16, torch.bfloat16)])
def test_gated_group_norm(n, group, types):
    to, tg, tout = types
    g = torch.Generator(device="cuda").manual_seed(n + group)
    rows = 5
    wide = torch.randn(rows, n + 8, generator=g, device="cuda").to(tg)
    o = torch.randn(rows, n, generator=g, device="cuda").to(to)
    w = torch.randn(n, generator=g, device="cuda").to(tg)
    for at in (0, 4, 8):                                # gates whose rows start on 16 bytes, and not
        gate = wide[:, at:at + n]
        for act in ("sigmoid", "silu"):
            got = ops.gated_group_norm(o, group, w, gate, act, 1e-5, tout)
            ref = o.double()
            if group:
                ref = ref.view(rows, -1, group)
                ref = (ref / torch.sqrt(ref.square().mean(-1, keepdim=True) + 1e-5)).view(rows, n)
            close(got, ref * w.double() * ACT[act](gate.double()), group)
    if n % 8 == 0 and group:                            # one gate value per 8 elements, no weight
        gate = wide[:, :n // 8].contiguous()
        ref = o.double().view(rows, -1, group)
        ref = (ref / torch.sqrt(ref.square().mean(-1, keepdim=True) + 1e-5)).view(rows, n) * torch.sigmoid(gate.double()).repeat_interleave(8, 1)
        close(ops.gated_group_norm(o, group, None, gate, "sigmoid", 1e-5, tout, gate_span=8), ref, group)


@pytest.mark.parametrize("n,group", [(184, 184), (192, 192), (192, 64), (256, 256), (256, 8), (264, 264), (264, 8), (272, 16)])
@pytest.mark.parametrize("rows", [3, 4095, 4096])
@pytest.mark.parametrize("dtype", [torch.float32, BF16])
def test_rows_around_the_shortest_that_are_taken_in_pieces(n, group, rows, dtype):
    g = torch.Generator(device="cuda").manual_seed(n + group)
    o, gate, w = torch.randn(rows, n, generator=g, device="cuda"), torch.randn(rows, n, generator=g, device="cuda").to(dtype), torch.rand(n, generator=g, device="cuda").to(dtype)
    ref = o.double().view(rows, -1, group)
    ref = (ref / torch.sqrt(ref.square().mean(-1, keepdim=True) + 1e-5)).view(rows, n)
    close(ops.gated_group_norm(o, group, w, gate, "silu", 1e-5, dtype), ref * w.double() * ACT["silu"](gate.double()), group)


@pytest.mark.parametrize("H,dv,parts", [(64, 64, 1), (8, 16, 4), (6, 8, 3), (32, 64, 8), (5, 7, 1), (16, 12, 2), (130, 64, 1), (23, 8, 1), (24, 8, 1), (3, 64, 1)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_ssd_output(H, dv, parts, dtype):
    g = torch.Generator(device="cuda").manual_seed(H * dv + parts)
    rows, n = 3, H * dv
    o, D = torch.randn(rows, n, generator=g, device="cuda"), torch.randn(H, generator=g, device="cuda")
    both = torch.randn(rows, 2 * n + 3, generator=g, device="cuda").to(dtype)
    w = torch.randn(n, generator=g, device="cuda").to(dtype)
    for x, z in ((both[:, :n], both[:, n:2 * n]), (both[:, 3:3 + n], both[:, 3 + n:])):
        v = (o.double() + D.double().repeat_interleave(dv) * x.double()) * torch.nn.functional.silu(z.double())
        size = (o.double().abs() + (D.double().repeat_interleave(dv) * x.double()).abs()) * torch.nn.functional.silu(z.double()).abs()
        r = 1.0 / torch.sqrt(v.view(rows, parts, -1).square().mean(-1, keepdim=True) + 1e-5)
        scale = r.expand(-1, -1, n // parts).reshape(rows, n) * w.double()
        got = ops.ssd_output(o, x, z, D, w, dv, parts, 1e-5)
        eps = 2.0 ** -24 * (n // parts + 32)
        assert ((got.double() - v * scale).abs() <= eps * size * scale.abs() + (2.0 ** -8 * (v * scale).abs() if dtype == torch.bfloat16 else 0) + 1e-30).all()
