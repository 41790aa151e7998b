"""Two host threads with operands of different sizes at once: kernels whose shared memory depends on the sizes."""
import threading

import numpy as np
import pytest
import torch

from qstream_b200.csrc import ops
from test_gpu_scan_chunks import cut, i32

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def attention(dh):
    slot, pos, table = i32([0] * 64), i32(range(64)), i32([0]).view(1, 1)
    q, k, v = torch.randn(64, dh).cuda(), torch.randn(1, 1, 64, dh).cuda(), torch.randn(1, 1, 64, 64).cuda()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    return lambda: ops.attention(q, 1, 1, dh, 0.1, 0, slot, pos, table, 64, k, v, status, v_head_dim=64, n_seq=1)


def delta(dk):
    T = 64
    q, k, v, g, beta = (torch.rand(T, n).cuda() * 0.1 for n in (dk, dk, 16, dk, 1))
    state, starts, slots, chunks = torch.zeros(1, 1, 16, dk, device="cuda"), i32([0, T]), i32([0]), cut([T])
    return lambda: ops.state_scan("delta", q, k, v, state, starts, slots, 1, 1, dk, 16, chunks=chunks, key_decay=g, token_weight=beta)


def experts(top):
    x, up, down = torch.randn(4, 64).to(BF).cuda(), torch.randn(16, 32, 64).to(BF).cuda(), torch.randn(16, 64, 32).to(BF).cuda()
    idx, wts, slots = i32(np.arange(top)).expand(4, top).contiguous(), torch.ones(4, top, device="cuda"), i32(range(4))
    return lambda: ops.moe_experts_indirect(x, up, down, idx, wts, slots, "silu")


@pytest.mark.parametrize("make,sizes", [(attention, (64, 256)), (delta, (36, 256)), (experts, (8, 16))])
def test_launches_of_two_threads_do_not_meet(make, sizes):
    """A kernel's limit of shared memory belongs to the process: a thread must not lower it between another's setting and its launch."""
    calls, failed, gate = [make(n) for n in sizes], [], threading.Barrier(2)
    torch.cuda.synchronize()

    def loop(call):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                gate.wait(timeout=60)
                for _ in range(3000):
                    call()
                torch.cuda.current_stream().synchronize()
        except Exception as e:                          # noqa: BLE001 - whatever it is, the other thread must end first
            failed.append(e)

    threads = [threading.Thread(target=loop, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not failed, failed
