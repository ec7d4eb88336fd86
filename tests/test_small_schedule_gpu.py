"""GPU test of the one-block schedule of small batches (small_schedule in
sw_strips.cu): batch sizes around its rounds of 1,024 pairs and its limit, with
pairs of every class -- A/C/G/T, raw bytes, no score, empty -- and both bins."""
import numpy as np
import pytest

from helpers import first_mismatches, oracle_batch

pytestmark = pytest.mark.gpu

DNA_BENCH = (3, -3, -6, -1)


@pytest.mark.parametrize("n", [1, 31, 1023, 1024, 1025, 4095, 4096, 4097])
def test_every_class_at_the_rounds(built, workloads, n):
    rng = np.random.default_rng(90 + n)
    b = workloads.PairBatch.concat([
        workloads.custom_dna(n - min(n - 1, 40), 91, 30, 200, 20, 120, related=0.8),
        workloads.custom_dna(min(n - 1, 40), 92, 560, 900, 520, 700, related=0.9)]) if n > 1 else workloads.plain_dna(1, 91)
    # raw bytes among the short pairs only: the int32 passes of 4 to 32 lanes give a
    # raw pair whose reverse pass has a second strip inside the band wrong begins
    raw = (rng.random(n) < 0.1) & (np.arange(n) < max(1, n - 40))
    for k in np.nonzero(raw)[0]:
        at = int(b.query_off[k])
        b.query[at] = rng.choice([ord("N"), ord("a")])
    none = np.nonzero(rng.random(n) < 0.05)[0]  # no symbol in common: score 0
    for k in none:
        b.query[b.query_off[k]:b.query_off[k + 1]] = ord("A")
        b.ref[b.ref_off[k]:b.ref_off[k + 1]] = ord("C")
    order = rng.permutation(n)
    b = b.subset(order)
    a = built.Aligner(0)
    got = a.align_batch(b, built.make_scoring(built.DNA, scores=DNA_BENCH))
    a.close()
    bad, count = first_mismatches(got, oracle_batch(b, 0, scores=DNA_BENCH))
    assert count == 0, bad


def test_protein_scores_change_between_calls(built, workloads):
    """The scores on the device follow the call's matrix, also when it changes in
    place and back."""
    b = workloads.protein(60, seed=93)
    a = built.Aligner(0)
    m = np.asarray(built.scoring.BLOSUM62, dtype=np.int16).copy()
    first = a.align_batch(b, built.make_scoring(built.PROTEIN, matrix=m, gaps=(-6, -1)))
    other = a.align_batch(b, built.make_scoring(built.PROTEIN, matrix=2 * m, gaps=(-6, -1)))
    again = a.align_batch(b, built.make_scoring(built.PROTEIN, matrix=m, gaps=(-6, -1)))
    a.close()
    assert np.array_equal(first, again) and not np.array_equal(first[:, 0], other[:, 0])
    assert np.array_equal(first, oracle_batch(b, 1, gaps=(-6, -1)))
