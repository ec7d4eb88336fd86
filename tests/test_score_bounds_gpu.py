"""GPU tests of the forward pass with score bounds (sw_bound.cu, the pruned rows of
sw_dual.cu; DNA batches of 40,000 pairs and more): bit-exact against the oracle at the
edges of strips, with equal best cells, repeats, long gaps and unrelated pairs in one
unit, at every two-pair width, for scorings that bound gaps weakly or not at all, and
with scores past int16."""
import numpy as np
import pytest

from helpers import first_mismatches, oracle_batch
from test_dual_steps_gpu import DNA_BENCH, _edges, _ties

pytestmark = pytest.mark.gpu


def _batch(workloads, seed):
    rng = np.random.default_rng(seed)
    refs, qs = _edges(0, rng)
    more = _ties(0, rng)
    refs, qs = refs + more[0], qs + more[1]
    for n in (100, 300, 700):  # a long gap on either side, a segment moved, a repeat
        a, b, c = ("".join(rng.choice(list("ACGT"), n)) for _ in range(3))
        refs += [a + b + c, a + c, a + b + c, a + a + b, a + "ACGT" * n, c + b + a]
        qs += [a + c, a + b + c, b + a, a, "ACGT" * (n // 2), a]
    return workloads.PairBatch.concat([
        workloads.PairBatch.from_strings(0, refs, qs), workloads.dna_throughput(150, seed=seed),
        workloads.mixed_dna(60, seed=seed + 1), workloads.custom_dna(150, seed + 2, 20, 700, 10, 400, related=0.5),
        workloads.PairBatch.from_strings(0, ["ACGTNNacgt" * 30, "AAAA", ""], ["ACGTNNACGT" * 20, "CCCC", "ACGT"])])


@pytest.mark.parametrize("width,scores", [(4, DNA_BENCH), (8, DNA_BENCH), (16, DNA_BENCH), (0, DNA_BENCH), (0, (1, 0, 0, 0)),
                                          (0, (2, 1, -3, -1)), (0, (3, -3, -1, -2)), (0, (5, -4, -30, 0)),
                                          (4, (100, -28, -60, -2))])
def test_many_pairs(built, workloads, width, scores):
    b = _batch(workloads, 91 + width)
    copies = -(-40_000 // b.n)
    a = built.Aligner(0, lane_group=width)
    got = a.align_batch(b.subset(np.tile(np.arange(b.n), copies)), built.make_scoring(built.DNA, scores=scores))
    st = a.stats()
    a.close()
    assert st["bin_dual"][0] == 1 and (st["reruns"] > 0) == (scores[0] == 100), st
    got = got.reshape(copies, b.n, 5)
    np.testing.assert_array_equal(got, np.broadcast_to(got[0], got.shape))
    bad, count = first_mismatches(got[0], oracle_batch(b, 0, scores=scores))
    assert count == 0, "%d mismatching pairs, first: %s" % (count, bad)
