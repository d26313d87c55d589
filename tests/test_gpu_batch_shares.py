"""Decode attention of large batches: three CTAs per SM and chunks of 256 positions (heads of 128, at most four q heads per kv
head, more than one round of CTAs).  Same comparison and tolerance as the smaller batches have: float64, 1e-5 where an output
of |v| < 6 carries about (positions + 130) roundings of 2^-24 of its terms' random sum."""
import pytest

import test_gpu_portions as portions
from test_gpu_portions import tb, torch  # noqa: F401  (fixtures)

pytestmark = pytest.mark.gpu

EDGES = [1, 2, 31, 32, 33, 255, 256, 257, 258, 511, 512, 513, 0, 1023, 1025, 64]


@pytest.mark.parametrize("heads,kv,lengths", [
    (32, 8, EDGES), (16, 8, EDGES + [2049, 0]), (8, 8, [4096] + EDGES), (12, 4, EDGES * 2), (3, 1, EDGES * 5), (32, 8, [4000] * 10), (32, 8, [1] * 64)])
def test_large_batches(torch, tb, heads, kv, lengths):  # noqa: F811
    portions.test_attention_of_unequal_sequences(torch, tb, heads, kv, 128, lengths)
