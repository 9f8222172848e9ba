"""A tensor-core group that gives up a wait leaves the digits of its transform
incomplete: the last stages' kernel then writes nothing, neither a transform's
output nor a ciphertext, and after the report the same calls are exact again."""
import numpy as np
import pytest

from hmpc_gb300 import _lib, lhe
from hmpc_gb300.comp import Queue, Tensor
from hmpc_gb300.moduli import MODULI

pytestmark = pytest.mark.gpu

KEY = [2, 4, 6, 8, 1, 3, 5, 7]
MARK = 0x5A5A5A5A


@pytest.mark.parametrize("name", ["q128", "q256"])
@pytest.mark.parametrize("log_n,batch", [(9, 5), (12, 3), (14, 2)])
def test_nothing_is_written_after_a_wait_that_ran_out(oracle, cpu_threads, name, log_n, batch):
    n = 1 << log_n
    queue = Queue(key=KEY)
    q, p = queue.modulus(MODULI[name]), queue.modulus(MODULI["p64"])
    oq, op = oracle.Modulus(MODULI[name]), oracle.Modulus(MODULI["p64"])
    q.set_plan(n, batch, radix_bits=0)
    x, m = queue.uniform(q, (batch,), n), queue.uniform(p, (batch,), n)
    key = lhe.Key(queue.uniform(q, (), n), queue.uniform(q, (), n))
    outs = [Tensor(q, (batch,), n) for _ in range(4)]

    def run():
        for t in outs:
            t.data.fill_(MARK)
        queue.nonce = [7, 7, 7]
        queue.ntt(x, out=outs[0])
        queue.ntt_centered_binomial(q, n, (batch,), 20, out=outs[1])
        queue.nonce = [7, 7, 7]
        lhe.enc(queue, key, m, q, out=lhe.Ciphertext(outs[2], outs[3]))

    _lib.call("hmpc_context_set_test_wait", queue.handle, 2048, 1)
    run()
    with pytest.raises(_lib.HmpcError) as err:
        queue.wait()
    assert err.value.code == 6  # HMPC_ERROR_TIMEOUT
    assert all((t.data == MARK).all().item() for t in outs)

    _lib.call("hmpc_context_set_test_wait", queue.handle, 0, 0)
    run()
    queue.wait()
    c0, c1, _ = oracle.lhe_enc(oq, op, n, batch, key.a.numpy(), key.b.numpy(), m.numpy(), False, KEY, [7, 7, 7],
                               threads=cpu_threads)
    refs = [oracle.ntt(oq, n, batch, src=x.numpy(), threads=cpu_threads),
            oracle.ntt(oq, n, batch, sampler="cbd", variance_x2=20, key=KEY, nonce=[7, 7, 7], threads=cpu_threads),
            c0, c1]
    assert all(np.array_equal(t.numpy(), r) for t, r in zip(outs, refs))
    queue.close()
