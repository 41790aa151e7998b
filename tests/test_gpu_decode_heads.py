"""Decode attention of query heads that share a key head (csrc/attention_decode.cu) against float64."""
import numpy as np
import pytest
import torch

from qstream_b200.csrc import attention_bf16

pytestmark = pytest.mark.gpu


def case(G, per, d, dv, lens, seed):
    """Query rows, pages of 64 keys in an order of their own, and the page table; all numbers bfloat16."""
    rng = np.random.default_rng(seed)
    bf = lambda *s: torch.tensor(rng.normal(size=s)).bfloat16()                                    # noqa: E731
    n_pages = [(n + 63) // 64 for n in lens]
    q, k, v = bf(len(lens), G * per, d), bf(sum(n_pages), G, 64, d), bf(sum(n_pages), G, 64, dv)
    order, table, at = rng.permutation(sum(n_pages)), -np.ones((len(lens), max(n_pages)), np.int32), 0
    for i, n in enumerate(n_pages):
        table[i, :n] = order[at:at + n]
        at += n
    return q, k, v, table


def run(q, k, v, table, lens, G, **opts):
    i32 = lambda x: torch.as_tensor(np.asarray(x), dtype=torch.int32).cuda()                       # noqa: E731
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    T, H, d = q.shape
    out = attention_bf16.decode(q.reshape(T, -1).cuda(), H, G, d, d ** -0.5, opts.pop("window", 0), i32(range(T)), i32([n - 1 for n in lens]), i32(table), 64,
                                k.cuda(), v.cuda(), max(lens), status, v_head_dim=v.shape[-1], out_dtype=torch.float32, **opts)
    assert int(status.item()) == 0
    return out.double().cpu().numpy().reshape(T, H, -1)


def plain(q, k, v, table, lens, G, window=0, softcap=0.0, chunk=0):
    """(result, bound of its error) in float64."""
    q, k, v = (x.double().numpy() for x in (q, k, v))
    T, H, d = q.shape
    want, bound = np.zeros((T, H, v.shape[-1])), np.zeros((T, H, 1))
    for t, n in enumerate(lens):
        first = max(0, n - window) if window else (n - 1) // chunk * chunk if chunk else 0
        pages = table[t, :(n + 63) // 64]
        for h in range(H):
            g = h // (H // G)
            kk, vv = (x[pages, g].reshape(-1, x.shape[-1])[first:n] for x in (k, v))
            s = kk @ q[t, h] / np.sqrt(d)
            size = np.abs(kk) @ np.abs(q[t, h]) / np.sqrt(d)
            s = softcap * np.tanh(s / softcap) if softcap else s
            p = np.exp(s - s.max())
            want[t, h] = p @ vv / p.sum()
            # a score is a sum of d products, a result one of up to 320 within a split and of the splits: each step at most 2^-23 of its terms;
            # errors of the scores move the weights by twice their size, the exponential and the cap add a few roundings
            bound[t, h] = 2.0 ** -23 * (2 * (d + 8) * size.max() + 320 + n / 256 + 16) * np.abs(vv).max()
    return want, bound


@pytest.mark.parametrize("per", [2, 3, 4, 5, 8])
@pytest.mark.parametrize("G,d,dv", [(2, 128, 128), (1, 64, 64), (3, 8, 8), (2, 40, 72), (1, 72, 24), (1, 136, 256), (1, 256, 192)])
def test_heads_that_share_a_key_head(per, G, d, dv):
    lens = [1, 16, 17, 63, 64, 65, 130, 256, 257, 513, 700]
    args = case(G, per, d, dv, lens, per * d + dv)
    for opts in (dict(), dict(window=100), dict(window=1), dict(softcap=2.5), dict(chunk=96)):
        got = run(*args, lens, G, **opts)
        want, bound = plain(*args, lens, G, **opts)
        assert (np.abs(got - want) <= bound).all(), (opts, (np.abs(got - want) / bound).max())


def test_each_head_has_its_own_result_however_many_share_the_key_head():
    lens = [300, 77]
    q, k, v, table = case(1, 7, 128, 128, lens, 5)
    whole = run(q, k, v, table, lens, 1)
    for h in (2, 3, 4, 5):                  # the first h heads alone: the same bits
        np.testing.assert_array_equal(run(q[:, :h].contiguous(), k, v, table, lens, 1), whole[:, :h])


def test_what_is_not_finite_stays_in_its_column_and_as_it_is():
    lens = [100]
    q, k, v, table = case(1, 4, 64, 64, lens, 6)
    v[table[0, 0], 0, 10, 3] = float("inf")
    v[table[0, 1], 0, 20, 5] = float("-inf")
    v[table[0, 1], 0, 30, 9] = float("nan")
    v[table[0, 1], 0, 50, 11] = float("inf")            # beyond the last key
    got = run(q, k, v, table, lens, 1)[0]
    assert (got[:, 3] == np.inf).all() and (got[:, 5] == -np.inf).all() and np.isnan(got[:, 9]).all()
    assert np.isfinite(np.delete(got, [3, 5, 9], axis=1)).all()
