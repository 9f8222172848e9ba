"""The CUDA-core transform at the edges of its tiles: one to ten tile bits
(and larger requests, which run ten), columns wider than a tile leaves room
for, degrees below one warp's tile, batches that leave the last block's tiles
unfilled, every producer -- against the oracle."""
import numpy as np
import pytest

from hmpc_gb300.comp import Queue

pytestmark = pytest.mark.gpu

KEY = [9, 8, 7, 6, 5, 4, 3, 2]
MODULI = {1: 0xFFF00001, 2: 0x8822D80623320001, 5: 0x92155E09E949EDD961C374C93DE4B90B9F220001,
          8: 0xCFF479B9B12CCF05AF55BCA0D7AE005D53E20D920B577D2785F3A1F156740001}


@pytest.mark.parametrize("limbs", sorted(MODULI))
@pytest.mark.parametrize("log_n,batch", [(2, 1), (2, 41), (3, 5), (6, 37), (10, 3), (11, 1), (12, 7)])
@pytest.mark.parametrize("tile_bits,col_bits", [(0, 4), (1, 0), (5, 6), (6, 2), (7, 3), (10, 3), (13, 5)])
def test_tile_edges(oracle, cpu_threads, limbs, log_n, batch, tile_bits, col_bits):
    n = 1 << log_n
    queue = Queue(key=KEY)
    q, ref = queue.modulus(MODULI[limbs]), oracle.Modulus(MODULI[limbs])
    for inverse in (False, True):
        if tile_bits * limbs <= 80:  # larger tiles of many limbs are not a plan
            q.set_plan(n, batch, inverse, 3, tile_bits, col_bits)
    x = queue.uniform(q, (batch,), n)
    y = queue.ntt(x)
    assert np.array_equal(y.numpy(), oracle.ntt(ref, n, batch, src=x.numpy(), threads=cpu_threads))
    assert np.array_equal(queue.intt(y, out=y).numpy(), x.numpy())
    for variance_x2 in (1, 64):
        nonce = queue.nonce
        z = queue.ntt_centered_binomial(q, n, (batch,), variance_x2)
        assert np.array_equal(z.numpy(), oracle.ntt(ref, n, batch, sampler="cbd", variance_x2=variance_x2, key=KEY,
                                                    nonce=nonce, threads=cpu_threads))
    nonce = queue.nonce
    z = queue.ntt_uniform(q, n, (batch,))
    assert np.array_equal(z.numpy(), oracle.ntt(ref, n, batch, sampler="uniform", key=KEY, nonce=nonce,
                                                threads=cpu_threads))
    queue.close()
