"""GPU test of the host entries around the sizes up to which they go through staging
(64 KB of inputs, 256 KB of results), for both result types."""
import numpy as np
import pytest

from helpers import first_mismatches, oracle_batch

pytestmark = pytest.mark.gpu

DNA_BENCH = (3, -3, -6, -1)


@pytest.mark.parametrize("int16", [False, True])
@pytest.mark.parametrize("n", [1, 7, 131, 132, 133, 134, 13_107, 13_108, 26_214, 26_215])
def test_results_on_both_sides_of_the_limits(built, workloads, n, int16):
    # 475 symbols and 16 bytes of offsets a pair: 64 KB at about 133 pairs
    b = workloads.plain_dna(n, seed=95) if n < 1000 else workloads.custom_dna(n, 95, 5, 40, 3, 30, related=0.7)
    a = built.Aligner(0)
    sc = built.make_scoring(built.DNA, scores=DNA_BENCH)
    got = [a.align_batch(b, sc, int16=int16), a.align_batch(b.subset(np.arange(n)[::-1]), sc, int16=int16)]
    a.close()
    exp = oracle_batch(b, 0, scores=DNA_BENCH)
    for g, e in ((got[0], exp), (got[1], exp[::-1])):
        bad, count = first_mismatches(np.asarray(g, dtype=np.int32), e)
        assert count == 0, bad
