"""What a dispatch takes from the server's pool is what it uses: an encryption
in the requests' own buffers three polynomials' words per plaintext, whatever
the transform's plan, and batched transforms in their own buffers nothing."""
import numpy as np
import pytest

from hmpc_gb300 import lhe, serving
from hmpc_gb300.comp import Queue, Tensor
from hmpc_gb300.moduli import MODULI

pytestmark = pytest.mark.gpu

KEY = [3, 1, 4, 1, 5, 9, 2, 6]
N = 1 << 10
COUNTS = (2, 1, 3)


@pytest.fixture()
def queue():
    q = Queue(key=KEY)
    yield q
    q.close()


def serve(queue, budget, submit):
    server = serving.Server(queue, memory_budget=budget, lanes=1, max_batch=len(COUNTS), batch_window_us=50000)
    queue.wait()
    assert None not in submit(server)
    server.drain()
    stats = server.stats()
    assert stats["failed"] == 0
    server.close()
    return stats


@pytest.mark.parametrize("tensor_cores", [False, True])
@pytest.mark.parametrize("counts", [COUNTS[:1], COUNTS])
def test_encryptions_in_a_pool_that_just_fits(queue, oracle, cpu_threads, tensor_cores, counts):
    q, p = queue.modulus(MODULI["q256"]), queue.modulus(MODULI["p64"])
    oq, op = oracle.Modulus(MODULI["q256"]), oracle.Modulus(MODULI["p64"])
    q.prepare(N)
    if tensor_cores:
        for polys in range(1, sum(counts) + 1):
            q.set_plan(N, polys, radix_bits=0)
    key = lhe.Key(queue.uniform(q, (), N), queue.uniform(q, (), N))
    work = [(queue.uniform(p, (c,), N), Tensor(q, (c,), N), Tensor(q, (c,), N), [c, 2, 3]) for c in counts]

    def submit(server):
        kid = server.add_key(q, p, key)
        queue.wait()
        return [server.submit_encrypt(kid, q, *w) for w in work]

    stats = serve(queue, 3 * q.limbs * N * sum(counts) * 4, submit)
    assert stats["dispatches"] == 1
    for x, c0, c1, nonce in work:
        r0, r1, _ = oracle.lhe_enc(oq, op, N, x.batch, key.a.numpy(), key.b.numpy(), x.numpy(), False, KEY, nonce,
                                   threads=cpu_threads)
        assert np.array_equal(c0.numpy(), r0) and np.array_equal(c1.numpy(), r1)


@pytest.mark.parametrize("shared", [False, True])
def test_transforms_without_a_pool(queue, oracle, cpu_threads, shared):
    """apart in one dispatch; into one buffer they would have to be gathered,
    which the pool has no room for: one after another"""
    q, oq = queue.modulus(MODULI["q192"]), oracle.Modulus(MODULI["q192"])
    q.prepare(N)
    xs = [queue.uniform(q, (2,), N) for _ in COUNTS]
    y = Tensor(q, (2,), N)
    ys = [y if shared else Tensor(q, (2,), N) for _ in COUNTS]
    stats = serve(queue, 256, lambda server: [server.submit_ntt(q, *w) for w in zip(xs, ys)])
    assert stats["dispatches"] == (len(COUNTS) if shared else 1)
    for x, out in list(zip(xs, ys))[-1 if shared else 0:]:
        assert np.array_equal(out.numpy(), oracle.ntt(oq, N, 2, src=x.numpy(), threads=cpu_threads))
