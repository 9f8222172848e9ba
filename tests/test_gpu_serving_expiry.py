"""A tensor-core transform of a serving dispatch that gives up a bounded wait:
its requests are reported as failed and their outputs left alone, and the lane's
next dispatches are exact again."""
import numpy as np
import pytest

from hmpc_gb300 import _lib, serving
from hmpc_gb300.comp import Queue, Tensor
from hmpc_gb300.moduli import MODULI

pytestmark = pytest.mark.gpu

MARK = 0x5A5A5A5A


@pytest.mark.parametrize("counts", [(2,), (1, 3)])
def test_failed_requests_and_a_usable_lane(oracle, cpu_threads, counts):
    queue = Queue(key=[8] * 8)
    q, oq = queue.modulus(MODULI["q192"]), oracle.Modulus(MODULI["q192"])
    n = 1 << 12
    q.prepare(n)
    q.set_plan(n, sum(counts), radix_bits=0)
    xs = [queue.uniform(q, (c,), n) for c in counts]
    ys = [Tensor(q, (c,), n) for c in counts]
    server = serving.Server(queue, lanes=1, max_batch=len(counts), batch_window_us=50000)
    for stall in (0, 1, 0):
        for y in ys:
            y.data.fill_(MARK)
        _lib.call("hmpc_context_set_test_wait", queue.handle, 2048 if stall else 0, stall)
        queue.wait()
        tickets = [server.submit_ntt(q, x, y) for x, y in zip(xs, ys)]
        server.drain()
        assert [server.poll(t)[0] for t in tickets] == [serving.FAILED if stall else serving.DONE] * len(counts)
        if not stall:
            for x, y in zip(xs, ys):
                assert np.array_equal(y.numpy(), oracle.ntt(oq, n, x.batch, src=x.numpy(), threads=cpu_threads))
        elif len(counts) == 1:  # several are gathered, and the scatter copies what is there
            assert (ys[0].data == MARK).all().item()
    server.close()
    queue.close()
