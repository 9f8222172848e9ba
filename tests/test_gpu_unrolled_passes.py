"""Passes of one and two limbs, unrolled for their number of stages: contiguous
passes of one to ten stages and the column passes that go with them, tensors
and samplers, polynomials of uneven degree -- against the oracle."""
import numpy as np
import pytest

from hmpc_gb300.batch import NttBatch
from hmpc_gb300.comp import Queue

pytestmark = pytest.mark.gpu

KEY = [1, 1, 2, 3, 5, 8, 13, 21]
MODULI = [0xFFF00001, 0x8822D80623320001]


@pytest.mark.parametrize("value", MODULI)
@pytest.mark.parametrize("tile_bits", range(1, 11))
@pytest.mark.parametrize("log_n,batch", [(10, 3), (15, 1)])
def test_every_number_of_stages(oracle, cpu_threads, value, tile_bits, log_n, batch):
    n = 1 << log_n
    queue = Queue(key=KEY)
    q, ref = queue.modulus(value), oracle.Modulus(value)
    x = queue.uniform(q, (batch,), n)
    want = oracle.ntt(ref, n, batch, src=x.numpy(), threads=cpu_threads)
    nonce = queue.nonce
    want_cbd = oracle.ntt(ref, n, batch, sampler="cbd", variance_x2=20, key=KEY, nonce=nonce, threads=cpu_threads)
    for col_bits in (1, 4):
        for inverse in (False, True):
            q.set_plan(n, batch, inverse, 3, tile_bits, col_bits)
        y = queue.ntt(x)
        assert np.array_equal(y.numpy(), want)
        assert np.array_equal(queue.intt(y).numpy(), x.numpy())
        queue.nonce = nonce
        assert np.array_equal(queue.ntt_centered_binomial(q, n, (batch,), 20).numpy(), want_cbd)
    queue.close()


@pytest.mark.parametrize("value", MODULI)
@pytest.mark.parametrize("inverse", [False, True])
def test_uneven_degrees(oracle, cpu_threads, value, inverse):
    queue = Queue(key=KEY)
    q, ref = queue.modulus(value), oracle.Modulus(value)
    degrees = [1 << k for k in (3, 15, 4, 10, 12, 13, 10)]
    xs = [queue.uniform(q, (), n) for n in degrees]
    batch = NttBatch(queue, q, degrees, inverse=inverse, autotune=False)
    for x, y, n in zip(xs, batch.run(xs), degrees):
        want = oracle.ntt(ref, n, 1, src=x.numpy(), inverse=inverse, threads=cpu_threads)
        assert np.array_equal(y.numpy(), want)
    assert batch.status() == 0
    batch.close()
    queue.close()
