"""The stream cipher at the edges of its tiles (512 elements, up to 16 limbs;
wider elements take the per-block kernel), both directions, against the oracle."""
import ctypes

import numpy as np
import pytest

from hmpc_gb300 import _lib
from hmpc_gb300.comp import Queue

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limbs", [1, 2, 3, 5, 6, 8, 9, 15, 16, 17, 33])
@pytest.mark.parametrize("elements", [1, 15, 511, 512, 513, 4096 + 257])
def test_cipher_edges(oracle, limbs, elements):
    import torch

    queue = Queue(key=[0] * 8)
    key, nonce = list(range(3, 11)), [5, 6, 7]
    planar = np.random.default_rng(limbs).integers(0, 2**32, size=(limbs, elements), dtype=np.uint64).astype(np.uint32)
    want = oracle.cipher_enc(key, nonce, planar)
    x = torch.from_numpy(planar.view(np.int32)).cuda()
    y = torch.full((limbs * elements + 8,), 7, dtype=torch.int32, device="cuda")
    z = torch.full((limbs * elements + 8,), 7, dtype=torch.int32, device="cuda")
    k, n = (ctypes.c_uint32 * 8)(*key), (ctypes.c_uint32 * 3)(*nonce)
    _lib.call("hmpc_cipher_enc", queue.handle, k, n, elements, limbs, x.data_ptr(), y.data_ptr())
    _lib.call("hmpc_cipher_dec", queue.handle, k, n, elements, limbs, y.data_ptr(), z.data_ptr())
    queue.wait()
    got = y.cpu().numpy().view(np.uint32)
    assert np.array_equal(got[:-8], want) and (got[-8:] == 7).all()
    back = z.cpu().numpy().view(np.uint32)
    assert np.array_equal(back[:-8], planar.reshape(-1)) and (back[-8:] == 7).all()
    queue.close()
