"""The end-to-end loop of bench.py: which buffer set holds the last step's
ciphertexts, after loops of any length one after another (each step encrypts
under a key of its own, so the set of the step before does not decrypt)."""
import pytest

import bench


@pytest.mark.parametrize("counts", [(3, 20), (3, 20, 215), (3, 20, 272), (5, 7, 8), (3, 1), (3, 4, 1)])
def test_the_last_steps_set(counts):
    sets = [{}, {}]
    key = 0

    def load(i):
        sets[i % 2]["message"] = i

    def encrypt(i):
        nonlocal key
        key += 1
        assert sets[i % 2]["message"] == i
        sets[i % 2]["ciphertext"] = (key, i)

    def read(i):
        assert sets[i % 2]["ciphertext"][1] == i  # not yet overwritten by a later step
        sets[i % 2]["host"] = sets[i % 2]["ciphertext"]

    for count in counts:
        last = bench.double_buffered(count, load, encrypt, read)
    assert sets[last]["host"] == (key, counts[-1] - 1)
