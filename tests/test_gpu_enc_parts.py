"""Key generation and encryption without a tensor-core plan: the transforms
run as parts of one set of passes where p has one or two limbs and q at least
72 bits, one after another otherwise.  Both sides of those limits, plaintexts
at the centring edges, odd batches and degrees, the nonce -- against the
oracle."""
import random

import numpy as np
import pytest

from hmpc_gb300 import lhe
from hmpc_gb300.comp import Queue, Tensor

pytestmark = pytest.mark.gpu

KEY = [2, 7, 1, 8, 2, 8, 1, 8]


def _prime(bits, step):
    """the largest prime below 2^bits that is 1 modulo `step`"""
    def is_prime(n):
        if any(n % f == 0 for f in (3, 5, 7, 11, 13, 17, 19, 23)):
            return False
        d, s = n - 1, 0
        while d % 2 == 0:
            d, s = d // 2, s + 1
        for a in (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37):
            x = pow(a, d, n)
            if x in (1, n - 1):
                continue
            for _ in range(s - 1):
                x = x * x % n
                if x == n - 1:
                    break
            else:
                return False
        return True

    n = ((1 << bits) - 2) // step * step + 1
    while not is_prime(n):
        n -= step
    return n


@pytest.mark.parametrize("q_bits,p_bits", [(71, 31), (72, 32), (72, 64), (96, 33), (128, 64), (160, 80), (250, 64),
                                           (256, 20), (288, 64), (288, 96)])
@pytest.mark.parametrize("log_n,batch", [(4, 5), (9, 1), (11, 3)])
def test_keys_and_encryption(oracle, cpu_threads, q_bits, p_bits, log_n, batch):
    n = 1 << log_n
    q_value, p_value = _prime(q_bits, 1 << 12), _prime(p_bits, 1 << 12)
    queue = Queue(key=KEY)
    queue.nonce = [0xFFFFFFF0, 0xFFFFFFFF, 7]  # the advance carries through the words
    q, p = queue.modulus(q_value), queue.modulus(p_value)
    oq, op = oracle.Modulus(q_value), oracle.Modulus(p_value)
    s, key = lhe.keygen(queue, q, p, n)
    s_ref, a_ref, b_ref, nonce = oracle.lhe_keygen(oq, op, n, KEY, [0xFFFFFFF0, 0xFFFFFFFF, 7])
    assert np.array_equal(s.numpy(), s_ref) and np.array_equal(key.b.numpy(), b_ref)
    assert np.array_equal(key.a.numpy(), a_ref) and queue.nonce == list(nonce)
    rng = random.Random(q_bits)
    canonical = [rng.choice([0, 1, p_value - 1, p_value >> 1, (p_value >> 1) + 1, rng.randrange(p_value)])
                 for _ in range(n * batch)]
    r = (1 << 32 * p.limbs) % p_value
    words = np.array([[(v * r % p_value >> 32 * j) & 0xFFFFFFFF for v in canonical] for j in range(p.limbs)],
                     dtype=np.uint32)
    x = Tensor.from_numpy(p, words, (batch,), n)
    for plaintext_ntt in (False, True):
        ct = lhe.enc(queue, key, x, q, plaintext_ntt=plaintext_ntt)
        c0, c1, nonce = oracle.lhe_enc(oq, op, n, batch, a_ref, b_ref, words, plaintext_ntt, KEY, nonce,
                                       threads=cpu_threads)
        assert np.array_equal(ct.c0.numpy(), c0) and np.array_equal(ct.c1.numpy(), c1)
        assert queue.nonce == list(nonce)
    queue.close()
