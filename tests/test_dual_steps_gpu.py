"""GPU tests of the two-pair int16x2 passes (sw_dual.cu): two rows a step in chunks of
4 or 8 steps, at every width, bit-exact against the oracle at the edges of lanes,
strips, row pairs and chunks, with halves of unlike height in one unit, and with equal
best cells in several strips and rows (each strip starts its maximum at the best of the
strips before it)."""
import numpy as np
import pytest

from helpers import first_mismatches, oracle_batch

pytestmark = pytest.mark.gpu

DNA_BENCH = (3, -3, -6, -1)
AA_GAPS = (-6, -1)
LETTERS = {0: "ACGT", 1: "ARNDCQEGHILKMFPSTWYV"}


def _edges(kind, rng):
    letters = list(LETTERS[kind])
    refs, qs = [], []
    for short in (1, 2, 3, 7, 8, 9, 15, 16, 17, 31, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 513):
        for extra in (0, 1, 2, 7, 8, 9, int(rng.integers(10, 400))):
            a = rng.choice(letters, short)
            b = np.concatenate([a.copy(), rng.choice(letters, extra)])
            hit = rng.integers(0, len(b), len(b) // 15)
            b[hit] = rng.choice(letters, len(hit))
            pair = ("".join(b), "".join(a))
            refs.append(pair[extra % 2])
            qs.append(pair[1 - extra % 2])
    return refs, qs


def _ties(kind, rng):
    letters = list(LETTERS[kind])
    refs, qs = [], []
    for gap in (0, 1, 30, 61, 64, 100, 250):
        seg = "".join(rng.choice(letters, 24))
        fill = lambda: "".join(rng.choice(letters, gap))  # noqa: E731
        many = fill().join([seg] * 4)
        refs += [many, seg, many + fill(), seg + fill() + seg]
        qs += [seg, many, many, many]
    return refs, qs


@pytest.mark.parametrize("kind,width", [(0, 4), (0, 8), (0, 16), (1, 16), (1, 32)])
def test_edges_and_ties(built, workloads, kind, width):
    rng = np.random.default_rng(71 + width)
    refs, qs = _edges(kind, rng)
    more = _ties(kind, rng)
    batch = workloads.PairBatch.from_strings(kind, refs + more[0], qs + more[1])
    a = built.Aligner(0, lane_group=width)
    sc = (built.make_scoring(built.DNA, scores=DNA_BENCH) if kind == 0 else
          built.make_scoring(built.PROTEIN, matrix=built.scoring.BLOSUM62, gaps=AA_GAPS))
    got = a.align_batch(batch, sc)
    st = a.stats()
    a.close()
    assert st["bin_dual"][0] == 1 and st["rev_dual"][0] == 1, st
    bad, count = first_mismatches(got, oracle_batch(batch, kind, scores=DNA_BENCH, gaps=AA_GAPS))
    assert count == 0, "%d mismatching pairs, first: %s" % (count, bad)
