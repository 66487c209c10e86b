"""The rule the device parse rests on, against the serial parse of the CPU
restatement: a pair of words is an event or a tag exactly when the first's top
bit is clear and the second's set, so that every such pair of a stream is one
and every other word outside a pair is skipped on its own."""
import numpy as np
import pytest

from oracle.lm import LMOracle


@pytest.fixture(scope="module")
def O():
    return LMOracle(9)


def resyncs(O, words):
    O.reset_clock()
    return O.histogram(np.asarray(words, np.uint32))[2]["resyncs"]


def test_top_bits_of_a_pair(O):
    for a in range(4):
        for b in range(4):
            out = resyncs(O, [a << 30, b << 30])
            assert out == (0 if a < 2 and b >= 2 else 1), (a, b)


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_streams(O, seed):
    rng = np.random.default_rng(seed)
    w = rng.integers(0, 1 << 32, 5001, dtype=np.uint32) & np.uint32(0xC0073F3F)
    top = w >> np.uint32(31)
    start = (top[:-1] == 0) & (top[1:] == 1)
    second = np.concatenate(([False], start))[:-1]
    assert resyncs(O, w) == int((~start & ~second).sum())
