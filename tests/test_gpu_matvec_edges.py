"""Matrix-vector products of one column (a Montgomery product each) and of
several (added up, reduced once), moduli at the top and the bottom of every limb
count, operands at the ends of the range -- against the oracle."""
import random

import numpy as np
import pytest

from hmpc_gb300.comp import Queue, Tensor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limbs", range(1, 10))
@pytest.mark.parametrize("edge", ["top", "bottom"])
@pytest.mark.parametrize("batch,rows,cols,n", [(1, 1, 1, 1), (3, 5, 1, 129), (2, 1, 2, 64), (1, 3, 3, 1), (2, 2, 7, 33)])
def test_matvec_edges(oracle, limbs, edge, batch, rows, cols, n):
    width = 32 * limbs
    value = (1 << width) - 5 if edge == "top" else (1 << (width - 32)) | (1 << 31) | 1
    queue = Queue(key=[0] * 8)
    q, ref = queue.modulus(value), oracle.Modulus(value)
    rng = random.Random(limbs * cols)

    def tensor(shape):
        count = int(np.prod(shape)) * n
        values = [rng.choice([0, 1, value - 1, value - 2, rng.randrange(value)]) for _ in range(count)]
        words = np.array([[(v >> (32 * j)) & 0xFFFFFFFF for v in values] for j in range(limbs)], dtype=np.uint32)
        return Tensor.from_numpy(q, words, shape, n)

    m, x = tensor((batch, rows, cols)), tensor((batch, cols))
    want = oracle.matvec(ref, batch, rows, cols, n, m.numpy(), x.numpy())
    assert np.array_equal(queue.matrix_vector_product(m, x).numpy(), want)
    queue.close()
