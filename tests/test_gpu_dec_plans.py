"""Decryption inside the inverse transform's passes in the tile shapes that a
tuner can choose: the inverse transform mod q ends and the transform mod p
begins on the same tiles, over two and three passes -- against the oracle."""
import numpy as np
import pytest

from hmpc_gb300 import lhe
from hmpc_gb300.comp import Queue
from hmpc_gb300.moduli import MODULI

pytestmark = pytest.mark.gpu

KEY = [5, 7, 7, 2, 1, 5, 6, 6]


@pytest.mark.parametrize("name", ["q128", "q256"])
@pytest.mark.parametrize("log_n,batch", [(7, 3), (12, 3), (14, 2), (16, 1)])
def test_decryption_in_set_shapes(oracle, cpu_threads, name, log_n, batch):
    n = 1 << log_n
    queue = Queue(key=KEY)
    q, p = queue.modulus(MODULI[name]), queue.modulus(MODULI["p64"])
    oq, op = oracle.Modulus(MODULI[name]), oracle.Modulus(MODULI["p64"])
    s = queue.ntt_centered_binomial(q, n, (), 1)
    ct = lhe.Ciphertext(queue.uniform(q, (batch,), n), queue.uniform(q, (batch,), n))
    for ntt_form in (False, True):
        want = oracle.lhe_dec(oq, op, n, batch, s.numpy(), ct.c0.numpy(), ct.c1.numpy(), ntt_form,
                              threads=cpu_threads)
        for radix_bits, tile_bits, col_bits in [(3, t, c) for t in (7, 8, 9, 10) for c in (2, 3, 4)] + [(2, 2, 1),
                                                                                                      (3, 12, 6)]:
            q.set_plan(n, batch, True, radix_bits=radix_bits, local_bits=tile_bits, col_bits=col_bits)
            assert np.array_equal(lhe.dec(queue, s, ct, p, plaintext_ntt=ntt_form).numpy(), want)
    queue.close()


@pytest.mark.parametrize("tile_bits,col_bits", [(7, 4), (9, 2)])
def test_batched_requests_in_set_shapes(oracle, cpu_threads, tile_bits, col_bits):
    """transforms and encryptions of one serving dispatch, in its shape's tiles"""
    from hmpc_gb300 import serving
    from hmpc_gb300.comp import Tensor

    n, counts = 1 << 13, (1, 2)
    queue = Queue(key=KEY)
    q, p = queue.modulus(MODULI["q160"]), queue.modulus(MODULI["p64"])
    oq, op = oracle.Modulus(MODULI["q160"]), oracle.Modulus(MODULI["p64"])
    q.prepare(n)
    q.set_plan(n, sum(counts), radix_bits=3, local_bits=tile_bits, col_bits=col_bits)
    key = lhe.Key(queue.uniform(q, (), n), queue.uniform(q, (), n))
    server = serving.Server(queue, lanes=1, max_batch=len(counts), batch_window_us=50000)
    kid = server.add_key(q, p, key)
    ntts = [(queue.uniform(q, (c,), n), Tensor(q, (c,), n)) for c in counts]
    encs = [(queue.uniform(p, (c,), n), Tensor(q, (c,), n), Tensor(q, (c,), n), [c, 1, 1]) for c in counts]
    queue.wait()
    for w in ntts:
        server.submit_ntt(q, *w)
    for w in encs:
        server.submit_encrypt(kid, q, *w)
    server.drain()
    assert server.stats()["dispatches"] == 2 and server.stats()["failed"] == 0
    for x, y in ntts:
        assert np.array_equal(y.numpy(), oracle.ntt(oq, n, x.batch, src=x.numpy(), threads=cpu_threads))
    for x, c0, c1, nonce in encs:
        r0, r1, _ = oracle.lhe_enc(oq, op, n, x.batch, key.a.numpy(), key.b.numpy(), x.numpy(), False, KEY, nonce,
                                   threads=cpu_threads)
        assert np.array_equal(c0.numpy(), r0) and np.array_equal(c1.numpy(), r1)
    server.close()
    queue.close()
