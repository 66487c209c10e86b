"""The local parse of the device listmode path: streams whose words take any
top bits (events, tags and lone words in any order), of lengths around the
runs, tiles and packets, against the serial parse of the CPU restatement."""
import numpy as np
import pytest

from oracle import lm
from oracle.lm import LMOracle

STAT_KEYS = ("words_used", "prompts", "delayed", "timetags", "tags", "invalid", "unmapped", "doi_other", "doi7",
             "resyncs", "frame_start", "duration", "terminated")
PACKET = lm.PACKET_WORDS


def wild(seed, n):
    """Random words with small fields and any top bits, some of them the halves
    of time, singles and other tags."""
    rng = np.random.default_rng(seed)
    w = rng.integers(0, 1 << 32, n, dtype=np.uint32)
    w &= np.uint32(0xC0073F3F)  # top bits, head pair, crystals below 64, DOI 0
    tags = rng.random(n) < 3e-2
    w = np.where(tags, rng.choice(np.array([0x80008000, 0xC0008001, 0x8000A002, 0x80000003], np.uint32), n), w)
    return w.astype(np.uint32)


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_every_in_sync_pair_is_an_event(seed):
    """A serial parse from a packet's first word reaches exactly the pairs
    whose first word has its top bit clear and whose second has it set."""
    w = wild(seed, 5000).tolist()
    starts, pos = [], 0
    while pos + 1 < len(w):
        in_sync = (w[pos] >> 31) == 0 and (w[pos + 1] >> 31) == 1
        if in_sync:
            starts.append(pos)
        pos += 2 if in_sync else 1
    assert starts == [p for p in range(len(w) - 1) if w[p] >> 31 == 0 and w[p + 1] >> 31 == 1]


@pytest.fixture(scope="module")
def pair():
    import hrrt_reconstruction_b200 as H
    O, D = LMOracle(9), H.Listmode(9)
    yield O, D
    D.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 127, 129, 511, 513, 4095, 4096, 4097, 4098, 8191,
                               PACKET - 1, PACKET, PACKET + 1, PACKET + 4098])
def test_any_words(pair, n):
    O, D = pair
    w = wild(n, n)
    for mode, flags in ((lm.PROMPTS_AND_DELAYED, 0), (lm.TRUES, 16), (lm.TRUES, 32), (lm.TRUES, 64)):
        O.reset_clock()
        D.reset_clock()
        so, do, sto = O.histogram(w, mode=mode)
        sd, dd, std = D.histogram(w, mode=mode, flags=flags)
        assert [sto[k] for k in STAT_KEYS] == [std[k] for k in STAT_KEYS]
        assert np.array_equal(so, sd)
        if mode == lm.PROMPTS_AND_DELAYED:
            assert np.array_equal(do, dd)
