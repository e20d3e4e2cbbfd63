"""CPU model of the words in which the interval-batched FP64 operator (csrc/sg_ibatch.cu) multiplies by t.

Every t that floor() can leave, down to the last place below one, has to come back from its two words exactly, and the
product with the largest combination must stay within 64 bits.
"""
import pytest

from test_ibatch_model import mul, s32, split, split_signed

NEAR_ONE = (1 << 62) - (1 << 30)


def split_fraction(v):
    return tuple(s32(w) for w in (split(v) if v >= NEAR_ONE else split_signed(v)))


@pytest.mark.parametrize("t", [0.0, 2.0 ** -62, 0.5, 1 - 2.0 ** -20, 1 - 2.0 ** -31, 1 - 2.0 ** -32, 1 - 2.0 ** -32 - 2.0 ** -53,
                               1 - 2.0 ** -33, 1 - 2.0 ** -50, 1 - 2.0 ** -53])
def test_words_of_t(t):
    v = int(t * 2 ** 62)
    h, l = split_fraction(v)
    assert (h << 31) + l == v
    # combinations stay below 2^62 in magnitude; what mul() drops is less than two units
    for y in (0, 1, -1, (1 << 62) - 1, -(1 << 62), 3 ** 39, -3 ** 39):
        assert abs((mul(split(y), (h, l), 0) << 62) - y * v) <= 2 << 62
