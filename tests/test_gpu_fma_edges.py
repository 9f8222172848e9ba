"""Products plus a sum at every width of access: all alignments of the planes,
lengths around a block of each width, in place, against exact integers."""
import random

import numpy as np
import pytest

from hmpc_gb300 import _lib
from hmpc_gb300.comp import Queue

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limbs", [1, 2, 4, 5, 8, 9])
@pytest.mark.parametrize("elements", [1, 2, 3, 4, 254, 255, 256, 257, 258, 1024, 1025, 1028])
@pytest.mark.parametrize("offset", [0, 1, 2])
def test_fma_edges(limbs, elements, offset):
    import torch

    q_value = (1 << 32 * limbs) - 5
    inverse = pow(1 << 32 * limbs, -1, q_value)
    rng = random.Random(elements)
    queue = Queue(key=[0] * 8)
    q = queue.modulus(q_value)
    values = [[rng.choice([0, 1, q_value - 1, rng.randrange(q_value)]) for _ in range(elements)] for _ in range(3)]
    expected = [(a * b * inverse + c) % q_value for a, b, c in zip(*values)]
    size = limbs * elements
    # the addend is overwritten by the result
    for shift in (0, offset):
        buffers = []
        for operand in values:
            words = np.array([[(v >> (32 * j)) & 0xFFFFFFFF for v in operand] for j in range(limbs)], dtype=np.uint32)
            buffer = torch.full((size + 8,), -1, dtype=torch.int32, device="cuda")
            at = shift if operand is values[0] else offset
            buffer[at:at + size] = torch.from_numpy(words.view(np.int32).reshape(-1)).cuda()
            buffers.append((buffer, at))
        a, b, d = (buffer.data_ptr() + 4 * at for buffer, at in buffers)
        _lib.call("hmpc_fma", queue.handle, q.handle, elements, a, b, d, d)
        queue.wait()
        got = buffers[2][0].cpu().numpy().view(np.uint32)
        planes = got[offset:offset + size].reshape(limbs, elements)
        assert [sum(int(planes[j, i]) << (32 * j) for j in range(limbs)) for i in range(elements)] == expected
        assert (got[:offset] == 0xFFFFFFFF).all() and (got[offset + size:] == 0xFFFFFFFF).all()
    queue.close()
