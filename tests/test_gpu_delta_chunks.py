"""The gated delta rule in chunks of up to 64 tokens (csrc/delta_chunks.cu) against a float64 walk."""
import numpy as np
import pytest
import torch

from qstream_b200.csrc import ops
from test_gpu_scan_chunks import cut, i32, r32

pytestmark = pytest.mark.gpu


def make(T, H, G, dk, dv, seed, fast):
    rng = np.random.default_rng(seed)
    q, k = (rng.normal(0, 1, (T, G, dk)) for _ in range(2))
    q, k = (r32(x / np.linalg.norm(x, axis=-1, keepdims=True)) for x in (q, k))
    v, beta = r32(rng.normal(0, 1, (T, H, dv))), r32(rng.uniform(0, 1, (T, H)))
    g = r32(rng.uniform(0, 1, (T, H, dk)) if fast else 1 - 10 ** rng.uniform(-5, -0.7, (T, H, dk)))
    if fast:
        g[T // 3] = 0.0
        beta[T // 2] = 1.0
    return q, k, v, g, beta


def walk(q, k, v, g, beta, S):
    H, G = v.shape[1], q.shape[1]
    o = np.zeros_like(v)
    for t in range(q.shape[0]):
        qt, kt = np.repeat(q[t], H // G, 0), np.repeat(k[t], H // G, 0)
        S = g[t][:, :, None] * S
        u = beta[t][:, None] * (v[t] - np.einsum("hkv,hk->hv", S, kt))
        S = S + kt[:, :, None] * u[:, None, :]
        o[t] = np.einsum("hkv,hk->hv", S, qt)
    return o, S


def run(q, k, v, g, beta, state, starts, slots, chunks):
    T, H = beta.shape
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x.reshape(T, -1))).float().cuda()       # noqa: E731
    return ops.state_scan("delta", dev(q), dev(k), dev(v), state, i32(starts), i32(slots), len(slots), H, q.shape[2], v.shape[2], chunks=chunks,
                          key_decay=dev(g), token_weight=dev(beta), qk_group=H // q.shape[1])


@pytest.mark.parametrize("H,G,dk,dv", [(2, 1, 128, 128), (2, 2, 64, 64), (1, 1, 256, 48), (4, 2, 36, 130), (2, 1, 7, 5), (1, 1, 65, 17), (2, 2, 130, 16)])
@pytest.mark.parametrize("fast", [False, True])
def test_chunks_against_the_walk(H, G, dk, dv, fast):
    for lens, size, tail in (([300, 1, 63, 64, 65], 64, 3), ([17], 64, 0), ([230, 101], 100, 0)):
        T = sum(lens)
        q, k, v, g, beta = make(T, H, G, dk, dv, dk + dv + T, fast)
        slots = list(range(1, len(lens) + 1))[::-1]
        S0 = r32(np.random.default_rng(T).normal(0, 1, (len(lens) + 2, H, dv, dk)))
        state = torch.from_numpy(S0).float().cuda()
        starts = np.concatenate([[0], np.cumsum(lens)])
        pad = lambda x: np.concatenate([x, np.ones((tail, *x.shape[1:]))])                        # noqa: E731
        o = run(*(pad(x) for x in (q, k, v, g, beta)), state, starts, slots, cut(lens, size)).double().cpu().numpy().reshape(T + tail, H, dv)
        assert not o[T:].any()
        state = state.double().cpu().numpy()
        for i in range(len(lens)):
            sl = slice(starts[i], starts[i + 1])
            ref, S = walk(q[sl], k[sl], v[sl], g[sl], beta[sl], S0[slots[i]].transpose(0, 2, 1))
            # unit vectors, step sizes and decays of at most one: the state does not grow, and a chunk's system has norm-one steps,
            # so errors add up like the roundings of sums over 64 tokens and dk channels: about sqrt(n) of 2^-24 each; four times that
            bound = 4 * 2.0 ** -24 * (np.sqrt(64) + np.sqrt(dk)) * np.sqrt(max(1, lens[i] / 16))
            assert np.linalg.norm(o[sl] - ref) <= bound * np.linalg.norm(ref), (lens, i, np.linalg.norm(o[sl] - ref) / np.linalg.norm(ref) / bound)
            assert np.linalg.norm(state[slots[i]].transpose(0, 2, 1) - S) <= bound * np.linalg.norm(S)
        np.testing.assert_array_equal(state[[0, len(lens) + 1]], S0[[0, len(lens) + 1]])


def test_what_is_not_finite_reaches_no_earlier_token():
    T, H, dk, dv = 150, 2, 32, 40
    q, k, v, g, beta = make(T, H, H, dk, dv, 3, False)
    v[90, 1, 3], k[100, 0, 5], q[110, 1, 2] = np.inf, np.nan, np.nan
    state = torch.zeros(1, H, dv, dk, device="cuda")
    o = run(q, k, v, g, beta, state, [0, T], [0], cut([T])).cpu().numpy().reshape(T, H, dv)
    assert np.isfinite(o[:90]).all() and np.isfinite(o[:100, 0]).all() and np.isfinite(o[90:110, 1, :3]).all()
    assert not np.isfinite(o[90, 1, 3]) and not np.isfinite(o[100, 0]).any() and not np.isfinite(o[110, 1]).any() and np.isfinite(o[111:, 1, :3]).all()


def test_operands_in_bfloat16_and_absent_values():
    """What the walk in order takes, the chunks take: bfloat16 q, k and v (exact in 32-bit: the same bits), and no values at all."""
    T, H, dk, dv = 200, 2, 40, 24
    q, k, v, g, beta = make(T, H, 1, dk, dv, 8, False)
    wide = torch.from_numpy(np.concatenate([x.reshape(T, -1) for x in (q, k, v)], 1)).to(torch.bfloat16).cuda()
    q, k, v = wide[:, :dk], wide[:, dk:2 * dk], wide[:, 2 * dk:]
    g, beta = (torch.from_numpy(x.reshape(T, -1)).float().cuda() for x in (g, beta))
    S0 = torch.randn(1, H, dv, dk, generator=torch.Generator().manual_seed(1)).cuda()

    def scan(q, k, v, chunks, **kw):
        state = S0.clone()
        o = ops.state_scan("delta", q, k, v, state, i32([0, T]), i32([0]), 1, H, dk, dv, chunks=chunks, key_decay=g, token_weight=beta, qk_group=H, **kw)
        return o, state

    for values in (v, None):
        low = scan(q, k, values, cut([T]))
        high = scan(q.float(), k.float(), v.float() if values is not None else torch.zeros(T, H * dv, device="cuda"), cut([T]))
        walked = scan(q, k, values, None)
        for a, b, c in zip(low, high, walked):
            assert torch.equal(a, b)
            assert (a - c).norm() <= 4 * 2.0 ** -24 * (np.sqrt(64) + np.sqrt(dk)) * np.sqrt(T / 16) * c.norm()
        alone = scan(q, k, values, None, want_output=False)
        assert alone[0] is None and torch.equal(alone[1], walked[1])


@pytest.mark.parametrize("dk", [40, 128, 130])
def test_very_small_values_are_held_whole(dk):
    """Values and a state around 2^-120, where a number's last bfloat16 term is cut."""
    T, H, dv, low = 150, 2, 40, 2.0 ** -120
    q, k, v, g, beta = make(T, H, H, dk, dv, 9, False)
    S0 = r32(np.random.default_rng(2).normal(0, 1, (1, H, dv, dk)))
    for vs in (v * low, 0 * v):
        state = torch.from_numpy(S0 * low).float().cuda()
        o = run(q, k, vs, g, beta, state, [0, T], [0], cut([T])).double().cpu().numpy().reshape(T, H, dv)
        ref, S = walk(q, k, vs, g, beta, (S0[0] * low).transpose(0, 2, 1))
        bound = 4 * 2.0 ** -24 * (np.sqrt(64) + np.sqrt(dk)) * np.sqrt(T / 16)
        for x, y in ((o, ref), (state.double().cpu().numpy()[0].transpose(0, 2, 1), S)):
            x, y = x / low, y / low
            assert np.linalg.norm(x - y) <= bound * np.linalg.norm(y) + 2.0 ** -149 / low * T * np.sqrt(y.size), np.linalg.norm(x - y) / np.linalg.norm(y)


@pytest.mark.parametrize("T", [70, 128])
@pytest.mark.parametrize("dk", [40, 128, 130])
def test_numbers_above_the_largest_bfloat16_stay_in_the_state(dk, T):
    """A channel that no token reads, writes or decays holds 3.4e38, which has no bfloat16 terms: it stays, and nothing else is touched."""
    H, dv, big = 2, 40, np.float32(3.4e38)
    q, k, v, g, beta = make(T, H, H, dk, dv, 13, False)
    q[:, :, 5], k[:, :, 5], g[:, :, 5] = 0.0, 0.0, 1.0
    S0 = r32(np.random.default_rng(4).normal(0, 1, (1, H, dv, dk)))
    S0[:, :, :, 5] = 0.0
    got = []
    for held in (0.0, big):
        S = S0.copy()
        S[0, 1, 7, 5] = held
        state = torch.from_numpy(S).float().cuda()
        got.append((run(q, k, v, g, beta, state, [0, T], [0], cut([T])).cpu().numpy(), state.cpu().numpy()))
    (o, state), (o_big, state_big) = got
    assert state_big[0, 1, 7, 5] == big
    state_big[0, 1, 7, 5] = 0.0
    assert np.isfinite(o_big).all() and np.isfinite(state_big).all()
    bound = 4 * 2.0 ** -24 * (np.sqrt(64) + np.sqrt(dk)) * np.sqrt(max(1, T / 16))        # as above: other sums of the same terms
    assert np.linalg.norm(o_big - o) <= bound * np.linalg.norm(o) and np.linalg.norm(state_big - state) <= bound * np.linalg.norm(state)
