"""A drain returns when the last request has finished, not at its timeout: many
short bursts, each drained, as the end of one falls anywhere in the drain."""
import time

import pytest

from hmpc_gb300 import serving
from hmpc_gb300.comp import Queue, Tensor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes", [1, 4])
def test_no_drain_sleeps_through_the_end(lanes):
    queue = Queue(key=[1] * 8)
    q = queue.modulus((1 << 64) - (1 << 32) + 1)
    n = 64
    q.prepare(n)
    x = queue.uniform(q, (), n)
    outs = [Tensor(q, (), n) for _ in range(lanes)]
    queue.wait()
    server = serving.Server(queue, lanes=lanes, max_batch=1)
    slowest = 0.0
    for _ in range(5000):
        for out in outs:
            server.submit_ntt(q, x, out)
        begin = time.perf_counter()
        server.drain(timeout_ms=5000)
        slowest = max(slowest, time.perf_counter() - begin)
    assert slowest < 4
    server.close()
    queue.close()
