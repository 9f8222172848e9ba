"""Decryption inside the inverse transform's passes: one pass and several, p of
one and two limbs (three take the separate cast), p above q, the result written
over the ciphertext it came from -- against the oracle."""
import numpy as np
import pytest

from hmpc_gb300 import lhe
from hmpc_gb300.comp import Queue, Tensor
from tests.test_gpu_enc_parts import _prime

pytestmark = pytest.mark.gpu

KEY = [1, 6, 1, 8, 0, 3, 3, 9]


@pytest.mark.parametrize("q_bits,p_bits", [(40, 63), (72, 32), (100, 64), (192, 64), (192, 31), (256, 64), (288, 96)])
@pytest.mark.parametrize("log_n,batch", [(2, 3), (4, 1), (8, 5), (9, 2), (10, 3), (12, 7)])
@pytest.mark.parametrize("ntt_form", [False, True])
def test_decryption_passes(oracle, cpu_threads, q_bits, p_bits, log_n, batch, ntt_form):
    n = 1 << log_n
    queue = Queue(key=KEY)
    q_value, p_value = _prime(q_bits, 1 << 13), _prime(p_bits, 1 << 13)
    q, p = queue.modulus(q_value), queue.modulus(p_value)
    oq, op = oracle.Modulus(q_value), oracle.Modulus(p_value)
    s = queue.ntt_centered_binomial(q, n, (), 1)
    ct = lhe.Ciphertext(queue.uniform(q, (batch,), n), queue.uniform(q, (batch,), n))
    want = oracle.lhe_dec(oq, op, n, batch, s.numpy(), ct.c0.numpy(), ct.c1.numpy(), ntt_form, threads=cpu_threads)
    assert np.array_equal(lhe.dec(queue, s, ct, p, plaintext_ntt=ntt_form).numpy(), want)
    for half in (ct.c0, ct.c1):
        if p.limbs > q.limbs:
            continue
        keep = half.data.clone()
        over = half.data.view(-1)[:p.limbs * n * batch].view(p.limbs, n * batch)
        out = lhe.dec(queue, s, ct, p, plaintext_ntt=ntt_form, out=Tensor(p, (batch,), n, over))
        assert np.array_equal(out.numpy(), want)
        half.data.copy_(keep)
    queue.close()
