"""The recurrences in chunks of up to 64 tokens (csrc/scan_chunks.cu) against a float64 walk, every form at its edges."""
import numpy as np
import pytest
import torch

from qstream_b200.csrc import ops

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


def r32(a):
    return np.asarray(a, dtype=np.float32).astype(np.float64)


def dev(a, dtype=torch.float32):
    return torch.from_numpy(np.ascontiguousarray(a)).to(dtype).cuda()


def i32(a):
    return torch.tensor(list(a), dtype=torch.int32).cuda()


def make(mode, T, H, G, dk, dv, seed, fast=False):
    """Operands of a mode: q, k [T, G, dk], v [T, H, dv], the decays and weights as the kernels take them, and as factors."""
    rng = np.random.default_rng(seed)
    q, k, v = r32(rng.normal(0, 1, (T, G, dk))), r32(rng.normal(0, 1, (T, G, dk))), r32(rng.normal(0, 1, (T, H, dv)))
    kw, b, u = {}, np.ones((T, H)), None
    if mode == "decay":
        d = r32(np.linspace(0.05 if fast else 0.9, 0.9995, H))
        kw = dict(head_decay=dev(d))
        a = np.broadcast_to(d[None, :, None], (T, H, dk))
    elif mode in ("gated", "ssd"):
        d = r32(rng.uniform(0, 1, (T, H)) if fast else 1 - 10 ** rng.uniform(-5, -0.5, (T, H)))
        if fast:
            d[T // 2] = 0.0                             # forgets everything
        less = r32(d - 1) if mode == "ssd" else d
        b = r32(rng.uniform(0.1, 2, (T, H)))
        kw = dict(token_decay=dev(less), token_weight=dev(b))
        a = np.broadcast_to((less + 1 if mode == "ssd" else d)[:, :, None], (T, H, dk))
    elif mode == "wkv":
        z = r32(rng.normal(1.0 if fast else -3.0, 1.5, (T, H, dk)))
        u = r32(rng.normal(0, 1, (H, dk)))
        kw = dict(decay_logits=dev(z.reshape(T, -1)), bonus=dev(u))
        a = np.exp(-np.exp(z))
    else:
        z = r32(rng.normal(-4.0 if fast else 1.0, 2.0, (T, H, dk)))
        kw = dict(decay_logits=dev(z.reshape(T, -1)), decay_power=1.0 if fast else 0.125)
        a = (1 / (1 + np.exp(-z))) ** kw["decay_power"]
    return q, k, v, a, b, u, kw


def walk(mode, q, k, v, a, b, u, S):
    """The recurrence in float64 from S [H, dk, dv]; and the same with every factor's absolute value: what roundings act on."""
    H, G = v.shape[1], q.shape[1]
    out = []
    for s, f in ((S, lambda x: x), (np.abs(S), np.abs)):
        o = np.zeros_like(v)
        for t in range(q.shape[0]):
            qt, kt = (np.repeat(f(x[t]), H // G, 0) for x in (q, k))
            kv = (b[t][:, None] * kt)[:, :, None] * f(v[t])[:, None, :]
            new = a[t][:, :, None] * s + kv
            o[t] = np.einsum("hkv,hk->hv", s + f(u)[:, :, None] * kv if mode == "wkv" else new, qt)
            s = new
        out += [o, s]
    return out


def cut(lens, size=64):
    starts, owners, row = [0], [0], 0
    for n in lens:
        starts += [row + min(n, at + size) for at in range(0, n, size)]
        row += n
        owners.append(len(starts) - 1)
    return i32(starts), i32(range(len(starts) - 1)), i32(owners), len(starts) - 1


def check(mode, lens, H, G, dk, dv, seed, fast=False, size=64, tail=0, dtype=torch.float32):
    T = sum(lens)
    real = dv - 1 if mode == "gated" else dv
    q, k, v, a, b, u, kw = make(mode, T, H, G, dk, real, seed, fast)
    q, k, v = (x.astype(np.float32) for x in (q, k, v))
    if dtype == torch.bfloat16:
        q, k, v = (torch.from_numpy(x).to(dtype).float().numpy() for x in (q, k, v))
    q, k, v = (x.astype(np.float64) for x in (q, k, v))
    pad = lambda x: np.concatenate([x.reshape(T, -1), np.ones((tail, x[0].size))])         # noqa: E731
    slots = [(3 * i + 1) % (len(lens) + 2) for i in range(len(lens))]
    assert len(set(slots)) == len(slots)
    S0 = r32(np.random.default_rng(seed + 1).normal(0, 1, (len(lens) + 2, H, dv, dk)))
    state = dev(S0)
    starts = np.concatenate([[0], np.cumsum(lens)])
    if tail:
        kw = {n: (torch.cat([x, torch.zeros((tail,) + x.shape[1:], device="cuda")]) if torch.is_tensor(x) and x.shape[0] == T else x) for n, x in kw.items()}
    o = ops.state_scan(mode, dev(pad(q), dtype), dev(pad(k), dtype), dev(pad(v), dtype), state, i32(starts), i32(slots), len(lens), H, dk, dv,
                       chunks=cut(lens, size), qk_group=H // G, **kw).double().cpu().numpy().reshape(T + tail, H, dv)
    assert not o[T:].any()
    state = state.double().cpu().numpy()
    for i, n in enumerate(lens):
        sl = slice(starts[i], starts[i + 1])
        vv = np.concatenate([v[sl], np.ones((n, H, 1))], 2) if mode == "gated" else v[sl]
        ref, S, mag, mag_S = walk(mode, q[sl], k[sl], vv, a[sl], b[sl], u, S0[slots[i]].transpose(0, 2, 1))
        # roundings on the way of any term: two sums over channels, one over a chunk's tokens, one per chunk, and four per decay (the
        # functions behind a decay are within two units of 2^-24 relative to an exponent of up to 16)
        rounds = 2 * dk + 3 * size + n // size + 4 * n * (16 if mode in ("wkv", "gla") else 1) + 16
        assert (np.abs(o[sl] - ref) <= rounds * EPS * mag + 1e-30).all(), np.max(np.abs(o[sl] - ref) / (EPS * mag + 1e-30))
        assert (np.abs(state[slots[i]].transpose(0, 2, 1) - S) <= rounds * EPS * mag_S + 1e-30).all()
        # and what is typical stays far below what is possible
        assert np.linalg.norm(o[sl] - ref) <= 4e-6 * np.linalg.norm(ref)
    free = [s for s in range(len(lens) + 2) if s not in slots]
    np.testing.assert_array_equal(state[free], S0[free])


SIZES = [(2, 1, 64, 64), (2, 2, 128, 128), (3, 1, 16, 70), (2, 2, 130, 129), (1, 1, 7, 5), (4, 2, 36, 63), (4, 1, 128, 64), (2, 2, 64, 200)]


@pytest.mark.parametrize("mode", ["decay", "wkv", "gated", "gla", "ssd"])
@pytest.mark.parametrize("H,G,dk,dv", SIZES)
def test_chunks_against_the_walk(mode, H, G, dk, dv):
    """Heads at the edges of the tiles (64 columns, 64 and 128 channels, slices of 32 and 64), one to many tokens per chunk, heads
    that share q and k, another state before, rows of nobody behind."""
    if mode != "ssd":
        G = H
    for lens, tail in (([300, 1, 63, 64, 65], 3), ([17], 0)):
        check(mode, lens, H, G, dk, dv + (mode == "gated"), H * dk + dv + tail, tail=tail)


@pytest.mark.parametrize("mode", ["decay", "wkv", "gated", "gla", "ssd"])
def test_chunks_that_forget_at_once_or_are_long_or_in_bfloat16(mode):
    check(mode, [200, 70], 2, 2, 48, 40 + (mode == "gated"), 5, fast=True)
    check(mode, [230, 101], 2, 2, 20, 24 + (mode == "gated"), 6, size=100)
    check(mode, [130], 4, 2 if mode == "ssd" else 4, 64, 64 + (mode == "gated"), 7, dtype=torch.bfloat16)


@pytest.mark.parametrize("mode", ["decay", "wkv", "gated", "gla", "ssd"])
def test_what_is_not_finite_reaches_no_earlier_token(mode):
    T, H, dk, dv = 150, 2, 32, 40
    q, k, v, a, b, u, kw = make(mode, T, H, H, dk, dv, 11)
    v[90, 1, 3], k[100, 0, 5], q[110, 0, 2] = np.inf, np.nan, -np.inf
    n = dv + (mode == "gated")
    state = torch.zeros(1, H, n, dk, device="cuda")
    o = ops.state_scan(mode, dev(q.reshape(T, -1)), dev(k.reshape(T, -1)), dev(v.reshape(T, -1)), state, i32([0, T]), i32([0]), 1, H, dk, n,
                       chunks=cut([T]), **kw).cpu().numpy().reshape(T, H, n)
    assert np.isfinite(o[:90]).all() and np.isfinite(o[:100, 0]).all() and np.isfinite(o[90:, 1, :3]).all()
    assert not np.isfinite(o[90, 1, 3]) and not np.isfinite(o[100, 0]).any() and not np.isfinite(o[110, 0]).any()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("mode", ["decay", "wkv", "gated", "gla", "ssd"])
def test_very_small_values_are_held_whole(mode, dtype):
    """Values and a state around 2^-120, where a number's last bfloat16 term is cut: outputs and state as near as for ordinary ones."""
    T, H, dk, dv, low = 100, 2, 40, 36, 2.0 ** -120
    q, k, v, a, b, u, kw = make(mode, T, H, H, dk, dv, 21)
    q, k, v = (torch.from_numpy(x).to(dtype).double().numpy() for x in (q, k, v))
    n = dv + (mode == "gated")
    S0 = r32(np.random.default_rng(2).normal(0, 1, (1, H, n, dk)))
    ones = np.ones((T, H, 1))
    for small_v in (True, False):                       # all of it, or the state alone beside values of zero
        vs = torch.from_numpy(v * low if small_v else 0 * v).to(dtype).double().numpy()
        state = dev(S0 * low)
        o = ops.state_scan(mode, dev(q.reshape(T, -1), dtype), dev(k.reshape(T, -1), dtype), dev(vs.reshape(T, -1), dtype), state, i32([0, T]), i32([0]), 1, H,
                           dk, n, chunks=cut([T]), **kw).double().cpu().numpy().reshape(T, H, n)[:, :, :dv]
        ref, S, _, _ = walk(mode, q, k, np.concatenate([vs, ones], 2) if mode == "gated" else vs, a, b, u, (S0[0] * low).transpose(0, 2, 1))
        got = state.double().cpu().numpy()[0].transpose(0, 2, 1)[:, :, :dv]
        for x, y in ((o, ref[:, :, :dv]), (got, S[:, :, :dv])):
            x, y = x / low, y / low
            assert np.linalg.norm(x - y) <= 4e-6 * np.linalg.norm(y) + 2.0 ** -149 / low * T * np.sqrt(y.size), np.linalg.norm(x - y) / np.linalg.norm(y)


def test_one_decay_per_head_over_many_chunks():
    """Fifteen chunks under constant decays, operands above zero: the decays' roundings are the same in every chunk and must not add up."""
    T, H, dk, dv = 900, 8, 64, 64
    rng = np.random.default_rng(31)
    q, k, v = (r32(rng.uniform(0, 1, (T, H, d))) for d in (dk, dk, dv))
    d = r32(np.linspace(0.9, 0.9995, H))
    state = torch.zeros(1, H, dv, dk, device="cuda")
    o = ops.state_scan("decay", dev(q.reshape(T, -1)), dev(k.reshape(T, -1)), dev(v.reshape(T, -1)), state, i32([0, T]), i32([0]), 1, H, dk, dv,
                       chunks=cut([T]), head_decay=dev(d)).double().cpu().numpy().reshape(T, H, dv)
    ref, S, _, _ = walk("decay", q, k, v, np.broadcast_to(d[None, :, None], (T, H, dk)), np.ones((T, H)), None, np.zeros((H, dk, dv)))
    # a term of the state passes two roundings per chunk, of the state and of the chunk's decay: the root of 30 times 0.29 of 2^-23 for the oldest, and
    # what the unit cuts off, 2^-23; the outputs pass up to 63 more, of the decays within a chunk
    assert np.linalg.norm(state.double().cpu().numpy()[0].transpose(0, 2, 1) - S) <= 3e-7 * np.linalg.norm(S)
    assert np.linalg.norm(o - ref) <= 4e-7 * np.linalg.norm(ref)
