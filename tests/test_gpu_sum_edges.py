"""Sums of residues plane by plane: every alignment of the planes, lengths
around the aligned middle and one block, the largest values, against exact
integers."""
import random

import numpy as np
import pytest

from hmpc_gb300 import _lib
from hmpc_gb300.comp import Queue, Tensor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limbs", [1, 2, 3, 4, 8, 9])
@pytest.mark.parametrize("elements", [1, 256, 257, 258, 259, 260, 1021, 70001])
@pytest.mark.parametrize("offset", [0, 1, 2, 3])
def test_sum_edges(limbs, elements, offset):
    import torch

    q_value = (1 << 32 * limbs) - 5
    rng = random.Random(elements)
    queue = Queue(key=[0] * 8)
    q = queue.modulus(q_value)
    out = Tensor(q, ())
    for values in ([q_value - 1] * elements, [rng.randrange(q_value) for _ in range(elements)]):
        words = np.array([[(v >> (32 * j)) & 0xFFFFFFFF for v in values] for j in range(limbs)], dtype=np.uint32)
        buffer = torch.full((limbs * elements + 8,), -1, dtype=torch.int32, device="cuda")
        buffer[offset:offset + limbs * elements] = torch.from_numpy(words.view(np.int32).reshape(-1)).cuda()
        _lib.call("hmpc_reduce", queue.handle, q.handle, 0, elements, buffer.data_ptr() + 4 * offset, out.ptr())
        got = out.numpy()
        assert sum(int(got[j, 0]) << (32 * j) for j in range(limbs)) == sum(values) % q_value
    queue.close()
