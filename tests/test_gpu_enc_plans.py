"""Encryption on the CUDA cores runs in the tile shape that is set for q's
transforms of that degree and batch: as many passes as the shape takes, and the
oracle's ciphertexts."""
import numpy as np
import pytest

from hmpc_gb300 import lhe
from hmpc_gb300.comp import Queue
from hmpc_gb300.moduli import MODULI

pytestmark = pytest.mark.gpu

KEY = [1, 4, 1, 4, 2, 1, 3, 5]


def passes(log_n, tile_bits, col_bits):
    rest = max(0, log_n - tile_bits)
    widest = max(1, tile_bits - col_bits)
    return 1 + -(-rest // widest)


@pytest.mark.parametrize("name", ["q160", "q256"])
@pytest.mark.parametrize("tile_bits,col_bits", [(5, 3), (7, 2), (10, 4)])
@pytest.mark.parametrize("log_n,batch", [(6, 3), (13, 2), (14, 1)])
def test_parts_in_the_set_shape(oracle, cpu_threads, name, tile_bits, col_bits, log_n, batch):
    n = 1 << log_n
    queue = Queue(key=KEY)
    q, p = queue.modulus(MODULI[name]), queue.modulus(MODULI["p64"])
    oq, op = oracle.Modulus(MODULI[name]), oracle.Modulus(MODULI["p64"])
    q.set_plan(n, batch, radix_bits=3, local_bits=tile_bits, col_bits=col_bits)
    key = lhe.Key(queue.uniform(q, (), n), queue.uniform(q, (), n))
    x = queue.uniform(p, (batch,), n)
    nonce = queue.nonce
    before = queue.launches
    ct = lhe.enc(queue, key, x, q)
    assert queue.launches - before == passes(log_n, tile_bits, col_bits) + 1
    c0, c1, _ = oracle.lhe_enc(oq, op, n, batch, key.a.numpy(), key.b.numpy(), x.numpy(), False, KEY, nonce,
                               threads=cpu_threads)
    assert np.array_equal(ct.c0.numpy(), c0) and np.array_equal(ct.c1.numpy(), c1)
    queue.close()
