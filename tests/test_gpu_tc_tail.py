"""The tensor-core forward transform's last stages on the CUDA cores: every
number of stages they can be (3 to 5), the smallest modulus that takes them and
the largest that does not, odd batches that leave the last block unfilled,
largest inputs, plain and as an encryption -- against the oracle."""
import numpy as np
import pytest

from hmpc_gb300 import lhe
from hmpc_gb300.comp import Queue, Tensor
from tests.test_gpu_enc_parts import _prime

pytestmark = pytest.mark.gpu

KEY = [3, 1, 4, 1, 5, 9, 2, 6]


@pytest.mark.parametrize("limbs", range(2, 9))
@pytest.mark.parametrize("short", [0, 14, 15])
@pytest.mark.parametrize("log_n,batch", [(8, 5), (9, 1), (9, 3), (10, 5), (11, 3), (12, 1), (13, 2), (14, 1)])
def test_tail(oracle, cpu_threads, limbs, short, log_n, batch):
    n = 1 << log_n
    # one bit below a full top byte where the digits of q / 2 would overflow
    q_value = _prime(32 * limbs - (short or 1), 1 << 15)
    queue = Queue(key=KEY)
    q, oq = queue.modulus(q_value), oracle.Modulus(q_value)
    q.set_plan(n, batch, False, radix_bits=0)
    x = queue.uniform(q, (batch,), n)
    words = x.numpy().copy()
    words[:, :n // 2] = np.array([[(q_value - 1) >> (32 * j) & 0xFFFFFFFF] for j in range(limbs)], dtype=np.uint32)
    x = Tensor.from_numpy(q, words, (batch,), n)
    assert np.array_equal(queue.ntt(x).numpy(), oracle.ntt(oq, n, batch, src=words, threads=cpu_threads))
    for variance_x2 in (1, 64):
        nonce = queue.nonce
        z = queue.ntt_centered_binomial(q, n, (batch,), variance_x2)
        assert np.array_equal(z.numpy(), oracle.ntt(oq, n, batch, sampler="cbd", variance_x2=variance_x2, key=KEY,
                                                    nonce=nonce, threads=cpu_threads))
    p_value = _prime(32, 1 << 13) if limbs == 2 else _prime(64, 1 << 13)
    p, op = queue.modulus(p_value), oracle.Modulus(p_value)
    msgs = queue.uniform(p, (batch,), n)
    key = lhe.Key(queue.uniform(q, (), n), queue.uniform(q, (), n))
    nonce = queue.nonce
    ct = lhe.enc(queue, key, msgs, q)
    c0, c1, _ = oracle.lhe_enc(oq, op, n, batch, key.a.numpy(), key.b.numpy(), msgs.numpy(), False, KEY, nonce,
                               threads=cpu_threads)
    assert np.array_equal(ct.c0.numpy(), c0) and np.array_equal(ct.c1.numpy(), c1)
    queue.wait()
    queue.close()
