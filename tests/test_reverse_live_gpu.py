"""GPU tests of the reverse pass's live rows (sw_dual.cu, launches of long DNA pairs: a strip
computes the rows from which the score can still be reached): bit-exact against the oracle for related pairs
with long gaps on either side, repeats, unrelated halves in one unit, and scorings that
make gaps cheap, dear or free, at every DNA width."""
import numpy as np
import pytest

from helpers import first_mismatches, oracle_batch
from test_dual_steps_gpu import DNA_BENCH
from test_score_bounds_gpu import _batch

pytestmark = pytest.mark.gpu


def _gapped(workloads, rng):
    refs, qs = [], []
    for n in (60, 130, 260, 540, 700):
        for gap in (1, 7, 40, 150, 400):
            a, b, c = ("".join(rng.choice(list("ACGT"), k)) for k in (n, n + gap // 3, gap))
            refs += [a + c + b, a + b, "".join(rng.choice(list("ACGT"), gap)) + a + c + b, a + c + b]
            qs += [a + b, a + c + b, a + b, a[: n // 2] + a[n // 2 + gap // 8:] + b]
    return workloads.PairBatch.from_strings(0, refs, qs)


@pytest.mark.parametrize("width", [4, 8, 16])
@pytest.mark.parametrize("scores", [DNA_BENCH, (1, -3, -3, -1), (5, -4, -30, -1), (3, -3, -1, -2), (2, -1, -2, -9), (1, 0, 0, 0)])
def test_live_rows(built, workloads, width, scores):
    rng = np.random.default_rng(101 + width)
    b = workloads.PairBatch.concat([_batch(workloads, 111), _gapped(workloads, rng),
                                    workloads.custom_dna(150, 113, 600, 1500, 520, 900, related=0.9)])
    a = built.Aligner(0)
    # plans apart, so that the long pairs are a launch of their own
    buckets = range(len(built.BUCKET_EDGES) + 1)
    a.set_tuning({(0, k, q): (1, 8) for k in (0, 1) for q in buckets},
                 {(0, k, q): (1, width if k else 24 - width if width == 16 else 16) for k in (0, 1) for q in buckets})
    got = a.align_batch(b, built.make_scoring(built.DNA, scores=scores))
    st = a.stats()
    a.close()
    assert st["rev_dual"][1] == 1 and st["rev_lanes"][1] == width and st["rev_lanes"][0] != width, st
    bad, count = first_mismatches(got, oracle_batch(b, 0, scores=scores))
    assert count == 0, "%d mismatching pairs, first: %s" % (count, bad)
