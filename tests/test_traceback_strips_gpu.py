"""GPU tests of the int16x2 traceback (trace_strips.cu): the oracle's operations at
the edges of strips, lanes and row pairs, across strips, for scorings at its
limits, and for batches that hold pairs for it and for the int32 kernel."""
import numpy as np
import pytest

from helpers import oracle_batch
from test_traceback_gpu import AA_GAPS, DNA_BENCH, _check

pytestmark = pytest.mark.gpu


def _identical_ends(workloads, kind, sizes, rng):
    """Segments of about the given lengths on either side: related pairs whose first
    and last symbols agree, a tenth of the rest changed, dropped or doubled."""
    letters = np.array(list("ACGT" if kind == 0 else "ARNDCQEGHILKMFPSTWYV"))
    refs, qs = [], []
    for n in sizes:
        for _ in range(3):
            a = rng.choice(letters, n)
            b = []
            for k, x in enumerate(a):
                u = rng.random() if 8 < k < n - 8 else 1.0
                if u < 0.04:
                    continue
                b.append(rng.choice(letters) if u < 0.08 else x)
                if u > 0.97 and u < 1.0:
                    b += list(rng.choice(letters, int(rng.integers(1, 40))))
            r, q = "".join(a), "".join(b)
            refs.append(r if len(refs) % 2 else q)
            qs.append(q if len(qs) % 2 else r)
    return workloads.PairBatch.from_strings(kind, refs, qs)


SIZES = (1, 2, 3, 4, 5, 31, 32, 33, 127, 128, 129, 255, 256, 257, 258, 511, 513, 700, 1100)


@pytest.mark.parametrize("kind", [0, 1])
def test_strip_and_lane_edges(built, workloads, aligner, kind):
    b = _identical_ends(workloads, kind, SIZES, np.random.default_rng(61 + kind))
    if kind == 0:
        _check(aligner, b, built.make_scoring(built.DNA, scores=DNA_BENCH), 0, scores=DNA_BENCH)
    else:
        sc = built.make_scoring(built.PROTEIN, matrix=built.scoring.BLOSUM62, gaps=AA_GAPS)
        _check(aligner, b, sc, 1, gaps=AA_GAPS)


# at and past its limits: equal gaps, gaps of 16 and 17 a symbol, scores 128 and 129
# apart, an opening cheaper than an extension
@pytest.mark.parametrize("scores", [(4, -2, -3, -3), (9, -9, -40, -16), (9, -9, -40, -17), (64, -64, -90, -2),
                                    (65, -64, -90, -2), (3, -3, -1, -2)])
def test_scorings_at_the_limits(built, workloads, aligner, scores):
    b = workloads.PairBatch.concat([_identical_ends(workloads, 0, SIZES, np.random.default_rng(63)),
                                    workloads.custom_dna(300, 64, 20, 700, 10, 400, related=0.6)])
    _check(aligner, b, built.make_scoring(built.DNA, scores=scores), 0, scores=scores)


def test_pairs_past_int16_beside_others(built, workloads, aligner):
    # 100 x length passes the score limit from 320 aligned symbols on
    scores = (100, -28, -60, -2)
    b = workloads.PairBatch.concat([_identical_ends(workloads, 0, (90, 300, 319, 320, 321, 400, 640),
                                                    np.random.default_rng(65)),
                                    workloads.custom_dna(200, 66, 200, 700, 150, 400, related=0.8)])
    res, _, _ = _check(aligner, b, built.make_scoring(built.DNA, scores=scores), 0, scores=scores)
    assert (res[:, 0] > 32_767).any() and (res[:, 0] < 20_000).any()
    assert np.array_equal(res, oracle_batch(b, 0, scores=scores))
