"""A dispatch of several requests works between the requests' own buffers, or
through one gathered buffer where its engine needs that (a plaintext modulus of
three limbs, a tensor-core plan): requests of one, two and three polynomials in
one batch, each as the oracle has it alone."""
import numpy as np
import pytest

from hmpc_gb300 import lhe, serving
from hmpc_gb300.comp import Queue, Tensor
from tests.test_gpu_enc_parts import _prime

pytestmark = pytest.mark.gpu

KEY = [4, 4, 4, 1, 2, 3, 4, 5]
COUNTS = (1, 3, 2)


@pytest.mark.parametrize("q_bits", [128, 250])
@pytest.mark.parametrize("p_bits", [32, 64, 96])
@pytest.mark.parametrize("log_n", [4, 11])
def test_encryptions_of_one_batch(oracle, cpu_threads, q_bits, p_bits, log_n):
    n = 1 << log_n
    queue = Queue(key=KEY)
    q_value, p_value = _prime(q_bits, 1 << 12), _prime(p_bits, 1 << 12)
    q, p = queue.modulus(q_value), queue.modulus(p_value)
    oq, op = oracle.Modulus(q_value), oracle.Modulus(p_value)
    q.prepare(n)
    key = lhe.Key(queue.uniform(q, (), n), queue.uniform(q, (), n))
    server = serving.Server(queue, lanes=1, max_batch=len(COUNTS), batch_window_us=50000)
    kid = server.add_key(q, p, key)
    work = [(queue.uniform(p, (c,), n), Tensor(q, (c,), n), Tensor(q, (c,), n), [0xFFFFFFFE, c, 9]) for c in COUNTS]
    queue.wait()
    for x, c0, c1, nonce in work:
        server.submit_encrypt(kid, q, x, c0, c1, nonce)
    server.drain()
    assert server.stats()["dispatches"] == 1 and server.stats()["failed"] == 0
    for x, c0, c1, nonce in work:
        r0, r1, _ = oracle.lhe_enc(oq, op, n, x.batch, key.a.numpy(), key.b.numpy(), x.numpy(), False, KEY, nonce,
                                   threads=cpu_threads)
        assert np.array_equal(c0.numpy(), r0) and np.array_equal(c1.numpy(), r1)
    server.close()
    queue.close()


@pytest.mark.parametrize("plan", [None, 0, 1])
@pytest.mark.parametrize("log_n", [10, 13])
def test_transforms_of_one_batch(oracle, cpu_threads, plan, log_n):
    n = 1 << log_n
    queue = Queue(key=KEY)
    q_value = _prime(159, 1 << 14)
    q, oq = queue.modulus(q_value), oracle.Modulus(q_value)
    q.prepare(n)
    if plan is not None:
        q.set_plan(n, sum(COUNTS), False, radix_bits=plan)
    server = serving.Server(queue, lanes=1, max_batch=len(COUNTS), batch_window_us=50000)
    work = [(queue.uniform(q, (c,), n), Tensor(q, (c,), n)) for c in COUNTS]
    work[1] = (work[1][0], work[1][0])  # one of them in place
    inputs = [x.numpy().copy() for x, _ in work]
    queue.wait()
    for x, y in work:
        server.submit_ntt(q, x, y)
    server.drain()
    assert server.stats()["dispatches"] == 1 and server.stats()["failed"] == 0
    for (_, y), x in zip(work, inputs):
        assert np.array_equal(y.numpy(), oracle.ntt(oq, n, y.batch, src=x, threads=cpu_threads))
    server.close()
    queue.close()
