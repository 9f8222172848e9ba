"""Casts between every pair of limb counts, moduli at the top and the bottom
of each, values at the ends of the range and around the centre, and the
conversions to and from Montgomery form, against exact integers."""
import random

import numpy as np
import pytest

from hmpc_gb300.comp import Queue, Tensor

pytestmark = pytest.mark.gpu


def _moduli(limbs):
    width = 32 * limbs
    return [(1 << width) - 5, (1 << (width - 32)) | (1 << 31) | 1]


def _tensor(q, values):
    words = np.array([[(v >> (32 * j)) & 0xFFFFFFFF for v in values] for j in range(q.limbs)], dtype=np.uint32)
    return Tensor.from_numpy(q, words, (len(values),))


def _values(t):
    words = t.numpy()
    return [sum(int(words[j, i]) << (32 * j) for j in range(words.shape[0])) for i in range(words.shape[1])]


@pytest.mark.parametrize("src_limbs", range(1, 10))
def test_cast_edges(src_limbs):
    queue = Queue(key=[0] * 8)
    rng = random.Random(src_limbs)
    for s_value in _moduli(src_limbs):
        s = queue.modulus(s_value)
        canonical = [0, 1, 2, s_value - 1, s_value - 2, s_value >> 1, (s_value >> 1) + 1, (s_value >> 1) - 1]
        canonical += [rng.randrange(s_value) for _ in range(301)]
        r_s = 1 << (32 * src_limbs)
        x = _tensor(s, [v * r_s % s_value for v in canonical])
        assert _values(queue.from_montgomery(x)) == canonical
        assert _values(queue.to_montgomery(_tensor(s, canonical))) == [v * r_s % s_value for v in canonical]
        centred = [v - s_value if v > s_value >> 1 else v for v in canonical]
        for dst_limbs in range(1, 10):
            for d_value in _moduli(dst_limbs):
                d = queue.modulus(d_value)
                want = [v % d_value * (1 << (32 * dst_limbs)) % d_value for v in centred]
                assert _values(queue.cast(x, d)) == want, (src_limbs, dst_limbs)
    queue.close()
