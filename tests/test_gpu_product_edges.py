"""The Montgomery product at the edges of its carry chains: moduli at the top
and the bottom of a limb count (even and odd counts), operands 0, 1, Q - 1,
single-limb and all-ones values, against exact integers."""
import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limbs", range(1, 10))
@pytest.mark.parametrize("edge", ["top", "bottom"])
def test_fma_edges(limbs, edge):
    from hmpc_gb300.comp import Queue, Tensor

    width = 32 * limbs
    q_value = (1 << width) - 5 if edge == "top" else (1 << (width - 32)) | (1 << 31) | 1
    rng = random.Random(limbs)
    special = [0, 1, 2, q_value - 1, q_value - 2, q_value >> 1, (q_value >> 1) + 1, 0xFFFFFFFF % q_value,
               ((1 << (width - 1)) - 1) % q_value]
    special += [((1 << 32) - 1 << 32 * j) % q_value for j in range(limbs)]
    triples = [(a, b, rng.choice(special)) for a in special for b in special]
    triples += [tuple(rng.randrange(q_value) for _ in range(3)) for _ in range(257)]
    queue = Queue(key=[0] * 8)
    q = queue.modulus(q_value)
    assert q.limbs == limbs

    def tensor(values):
        words = np.array([[(v >> (32 * j)) & 0xFFFFFFFF for v in values] for j in range(limbs)], dtype=np.uint32)
        return Tensor.from_numpy(q, words, (len(values),))

    d = queue.fma(*(tensor(column) for column in zip(*triples))).numpy()
    r_inv = pow(1 << width, -1, q_value)
    got = [sum(int(d[j, i]) << (32 * j) for j in range(limbs)) for i in range(len(triples))]
    assert got == [(a * b * r_inv + c) % q_value for a, b, c in triples]
