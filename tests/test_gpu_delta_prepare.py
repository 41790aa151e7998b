"""What comes before the gated delta rule (csrc/delta.cu): channels in pieces of eight, against float64 and the general kernel."""
import numpy as np
import pytest
import torch

from qstream_b200.csrc import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("G,H,dk,dv,taps", [(1, 1, 8, 8, 2), (2, 4, 16, 24, 3), (3, 3, 32, 40, 4), (1, 2, 64, 64, 4), (2, 2, 128, 128, 4), (1, 3, 256, 16, 2),
                                            (5, 5, 128, 8, 3)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T", [7, 600])                 # several blocks to a token, and one
def test_pieces_against_float64_and_the_general_kernel(G, H, dk, dv, taps, dtype, T):
    rng = np.random.default_rng(G * dk + dv + T)
    nq, nv = G * dk, H * dv
    C = 2 * nq + nv
    f32 = lambda x: torch.tensor(x).float().cuda()                                                 # noqa: E731
    low = lambda x: torch.tensor(x).to(dtype).cuda()                                               # noqa: E731
    i32 = lambda x: torch.as_tensor(x, dtype=torch.int32).cuda()                                   # noqa: E731
    x, w, held = low(rng.normal(0, 1, (T, C))), low(rng.normal(0, 1, (C, taps))), low(rng.normal(0, 1, (3, taps - 1, C)))
    a, b, a_log = f32(rng.normal(0, 3, (T, H * dk))), f32(rng.normal(0, 2, (T, H))), f32(rng.uniform(-3, 1, H))
    a[0, 0], a[1, 1] = 200.0, -200.0
    # two sequences, the first from position 4 on (its predecessors are held), a row of nobody at the end
    n = T // 2
    slot, pos = [2] * n + [0] * (T - 1 - n) + [-1], [*range(4, 4 + n), *range(T - 1 - n), 0]
    held[0] = 0                                         # a sequence's first tokens follow zeros
    conv = [w[:nq], w[nq:2 * nq], w[2 * nq:]]

    def run(x, a, taps_of):
        return ops.delta_prepare(x[:, :nq], x[:, nq:2 * nq], x[:, 2 * nq:C], *taps_of, held, a, b, a_log, i32(slot), i32(pos), G, H, dk, dv, dk ** -0.5, 1e-6)

    got = run(x, a, [c.contiguous() for c in conv])
    shifted = torch.zeros(T * H * dk + 1, device="cuda")[1:].view(T, H * dk)        # decays off the 16-byte boundary: the general kernel
    shifted.copy_(a)
    general = run(x, shifted, [c.contiguous() for c in conv])
    xd, wd, hd = (t.double().cpu().numpy() for t in (x, w, held))
    y = np.zeros((T, C))
    size = np.zeros((T, C))
    for t in range(T - 1):
        first = 0 if t < n else n
        for j in range(taps):
            src = xd[t - j] if t - j >= first else hd[slot[t], taps - 1 - (j - (t - first))]
            y[t] += wd[:, taps - 1 - j] * src
            size[t] += np.abs(wd[:, taps - 1 - j] * src)
    y, u = y / (1 + np.exp(-y)), 2.0 ** -23
    qk = y[:, :2 * nq].reshape(T, 2 * G, dk)
    norm = np.sqrt((qk ** 2).sum(-1, keepdims=True) + 1e-6)
    unit = (qk / norm).reshape(T, -1)
    near = (8 * size[:, :2 * nq].reshape(T, 2 * G, dk).max(-1, keepdims=True) / norm + dk / 8 + 16) * u * np.ones((1, 1, dk))
    near = near.reshape(T, -1)                          # a sum's roundings over the vector's length, and those of the length itself
    decay = np.exp(-np.exp(np.repeat(a_log.double().cpu().numpy(), dk)) * np.logaddexp(0, a.double().cpu().numpy()))
    decay[T - 1] = 1.0
    step = 1 / (1 + np.exp(-b.double().cpu().numpy()))
    step[T - 1] = 0.0
    want = (unit[:, :nq] * dk ** -0.5, unit[:, nq:], y[:, 2 * nq:], decay, step)
    bound = (near[:, :nq] * dk ** -0.5, near[:, nq:], 8 * u * size[:, 2 * nq:] + u * 8 * np.abs(y[:, 2 * nq:]), 64 * u, 8 * u)
    for g, r, ref, near in zip(got, general, want, bound):
        g, r = g.double().cpu().numpy(), r.double().cpu().numpy()
        assert (np.abs(g - ref) <= near + 1e-30).all(), (np.abs(g - ref) / (near + 1e-30)).max()
        assert (np.abs(g - r) <= 2 * near + 1e-30).all()
