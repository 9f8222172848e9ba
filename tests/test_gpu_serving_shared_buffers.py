"""Requests of one dispatch that share buffers: the same transform submitted
several times, a result over another request's input, two results in one
buffer.  The dispatch reads every input before it writes a result and the
results follow in the requests' order."""
import numpy as np
import pytest

from hmpc_gb300 import lhe, serving
from hmpc_gb300.comp import Queue, Tensor
from hmpc_gb300.moduli import MODULI

pytestmark = pytest.mark.gpu

KEY = [9, 8, 7, 6, 5, 4, 3, 2]


@pytest.fixture()
def queue():
    q = Queue(key=KEY)
    yield q
    q.close()


def run(queue, requests, kid=None):
    """requests: lists of submit_ntt's or submit_encrypt's arguments, as one dispatch"""
    server = serving.Server(queue, lanes=1, max_batch=len(requests), batch_window_us=50000)
    if kid is not None:
        key_id = server.add_key(*kid)
    queue.wait()
    for r in requests:
        server.submit_ntt(*r) if kid is None else server.submit_encrypt(key_id, *r)
    server.drain()
    stats = server.stats()
    assert stats["dispatches"] == 1 and stats["failed"] == 0
    server.close()


@pytest.mark.parametrize("name", ["q128", "q256"])
@pytest.mark.parametrize("log_n", [8, 13, 16])
def test_transforms_that_share_buffers(queue, oracle, cpu_threads, name, log_n):
    q, oq = queue.modulus(MODULI[name]), oracle.Modulus(MODULI[name])
    n = 1 << log_n
    q.prepare(n)
    x, w = queue.uniform(q, (2,), n), queue.uniform(q, (1,), n)
    one = Tensor(q, (1,), n, x.data.view(-1)[:q.limbs * n].view(q.limbs, n))  # the first words of x
    y = Tensor(q, (2,), n)
    references = {}
    for t in (x, w):
        references[t] = oracle.ntt(oq, n, t.batch, src=t.numpy(), threads=cpu_threads)
    kept = x.data.view(-1)[q.limbs * n:].clone()
    # four times the same, and w's transform over the first half of x's words
    run(queue, [(q, x, y)] * 4 + [(q, w, one)])
    assert np.array_equal(y.numpy(), references[x])
    assert np.array_equal(one.numpy(), references[w])
    assert (x.data.view(-1)[q.limbs * n:] == kept).all().item()


@pytest.mark.parametrize("log_n", [8, 13])
def test_encryptions_into_one_buffer(queue, oracle, cpu_threads, log_n):
    q, p = queue.modulus(MODULI["q160"]), queue.modulus(MODULI["p64"])
    oq, op = oracle.Modulus(MODULI["q160"]), oracle.Modulus(MODULI["p64"])
    n = 1 << log_n
    q.prepare(n)
    key = lhe.Key(queue.uniform(q, (), n), queue.uniform(q, (), n))
    x = [queue.uniform(p, (c,), n) for c in (1, 2, 2)]
    c0, c1 = Tensor(q, (2,), n), Tensor(q, (2,), n)
    # the second request's message ends under the first one's c1: read before it is written
    both = x[1].data.new_empty(q.limbs * n)
    both[:x[1].data.numel()] = x[1].data.view(-1)
    x[1] = Tensor(p, (2,), n, both[:x[1].data.numel()].view(p.limbs, 2 * n))
    first = (Tensor(q, (1,), n), Tensor(q, (1,), n, both.view(q.limbs, n)))
    refs = [oracle.lhe_enc(oq, op, n, t.batch, key.a.numpy(), key.b.numpy(), t.numpy(), False, KEY, [i, 5, 6],
                           threads=cpu_threads) for i, t in enumerate(x)]
    run(queue, [(q, x[0], *first, [0, 5, 6]), (q, x[1], c0, c1, [1, 5, 6]), (q, x[2], c0, c1, [2, 5, 6])],
        (q, p, key))
    assert np.array_equal(first[0].numpy(), refs[0][0]) and np.array_equal(first[1].numpy(), refs[0][1])
    assert np.array_equal(c0.numpy(), refs[2][0]) and np.array_equal(c1.numpy(), refs[2][1])
