"""GPU tests of the banded traceback (trace_band in trace_strips.cu, DNA calls of 12,000
pairs and more): the oracle's operations at the edges of strips, lanes, row pairs and
chunks, for narrow and full bands, tied paths, scorings at its limits and pairs past
them, and scores that are not their segment's refused."""
import numpy as np
import pytest

from test_traceback_gpu import DNA_BENCH, _check
from test_traceback_strips_gpu import _identical_ends

pytestmark = pytest.mark.gpu

SIZES = (1, 2, 3, 4, 5, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 129, 300, 700, 2040, 2047, 2049)


def _batch(workloads):
    tied = workloads.PairBatch.from_strings(
        0, ["A" * n for n in (40, 200, 333)] + ["ACGT" * 60, "AC" * 50 + "G" * 70 + "AC" * 50],
        ["A" * n for n in (57, 150, 333)] + ["ACGT" * 21 + "TTTTTTT" + "ACGT" * 30, "AC" * 100])
    return workloads.PairBatch.concat([
        _identical_ends(workloads, 0, SIZES, np.random.default_rng(81)), tied,
        workloads.custom_dna(400, 82, 20, 700, 10, 400, related=0.6),
        workloads.PairBatch.from_strings(0, ["ACGTNNacgt" * 30, "AAAA", ""], ["ACGTNNACGT" * 20, "CCCC", "ACGT"])])


# equal gaps; wide ones of 16 a symbol; 128 between match and mismatch (segments past the
# band kernel's values among them); an opening cheaper than an extension (int32 kernel)
@pytest.mark.parametrize("scores", [DNA_BENCH, (4, -2, -3, -3), (9, -9, -40, -16), (64, -64, -90, -2), (1, 0, 0, 0),
                                    (3, -3, -1, -2)])
def test_many_pairs(built, workloads, aligner, scores):
    b = _batch(workloads)
    sc = built.make_scoring(built.DNA, scores=scores)
    res, ops, off = _check(aligner, b, sc, 0, scores=scores)
    copies = -(-12_000 // b.n)
    many = np.tile(res, (copies, 1))
    got, got_off = aligner.traceback_batch(b.subset(np.tile(np.arange(b.n), copies)), sc, many)
    np.testing.assert_array_equal(np.diff(got_off), np.tile(np.diff(off), copies))
    np.testing.assert_array_equal(got, np.tile(ops, copies))


@pytest.mark.parametrize("by", [-30, -1, 1, 40, 2**31 - 1])
def test_other_scores_refused(built, workloads, aligner, by):
    b = workloads.dna_throughput(12_000, seed=83)
    sc = built.make_scoring(built.DNA, scores=DNA_BENCH)
    res = np.array(aligner.align_batch(b, sc))
    k = int(np.argmax(res[:, 0] > 300))
    res[k, 0] = by if by > 1000 else res[k, 0] + by
    with pytest.raises(built.GbswError):
        aligner.traceback_batch(b, sc, res)
