"""GPU tests of the strip-parallel int16x2 passes (sw_strips.cu, the automatic plan
of batches of up to a few thousand pairs): bit-exact against the oracle at the
edges of strips, lanes and row pairs, with 4 and 8 columns a lane, with more
strips than edge buffers, and with scores past int16."""
import numpy as np
import pytest

from helpers import first_mismatches, oracle_batch

pytestmark = pytest.mark.gpu

DNA_BENCH = (3, -3, -6, -1)
AA_GAPS = (-6, -1)


def _check(got, exp):
    bad, count = first_mismatches(got, exp)
    assert count == 0, "%d mismatching pairs, first: %s" % (count, bad)


def _pairs(workloads, kind, shorts, rng):
    """For each length: related pairs with the shorter side that long, either role,
    the longer side equal, one longer and up to 300 longer."""
    letters = list("ACGT" if kind == 0 else "ARNDCQEGHILKMFPSTWYV")
    refs, qs = [], []
    for short in shorts:
        for extra in (0, 1, int(rng.integers(2, 300))):
            a = rng.choice(letters, short)
            b = np.concatenate([a.copy(), rng.choice(letters, extra)])
            hit = rng.integers(0, len(b), max(1, len(b) // 15))
            b[hit] = rng.choice(letters, len(hit))
            r, q = "".join(b), "".join(a)
            refs.append(r if extra % 2 else q)
            qs.append(q if extra % 2 else r)
    return workloads.PairBatch.from_strings(kind, refs, qs)


def _align(built, batch, kind):
    sc = (built.make_scoring(built.DNA, scores=DNA_BENCH) if kind == 0 else
          built.make_scoring(built.PROTEIN, matrix=built.scoring.BLOSUM62, gaps=AA_GAPS))
    a = built.Aligner(0)
    got = a.align_batch(batch, sc)
    st = a.stats()
    a.close()
    return got, st


@pytest.mark.parametrize("kind", [0, 1])
def test_strip_and_lane_edges(built, workloads, kind):
    # 4 columns a lane: 128-column halves, 256-column strips
    batch = _pairs(workloads, kind, (1, 2, 3, 4, 5, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1023, 1025),
                   np.random.default_rng(41 + kind))
    got, st = _align(built, batch, kind)
    assert st["bin_lanes"][0] == 128 and st["reruns"] == 0, st
    _check(got, oracle_batch(batch, kind, scores=DNA_BENCH, gaps=AA_GAPS))


@pytest.mark.parametrize("n", [1, 2, 5])
def test_few_pairs(built, workloads, n):
    batch = workloads.long_dna(n, seed=43)
    got, _ = _align(built, batch, 0)
    _check(got, oracle_batch(batch, 0, scores=DNA_BENCH))


def test_eight_columns_and_reused_edge_buffers(built, workloads):
    # enough long pairs for 8 columns a lane (512-column strips), and more strips
    # than edge buffers, among them the widths around one and two strips
    batch = workloads.PairBatch.concat([
        workloads.custom_dna(2900, 44, 1100, 1500, 1030, 1400, related=0.8),
        _pairs(workloads, 0, (511, 512, 513, 1023, 1024, 1025, 1400), np.random.default_rng(45))])
    got, _ = _align(built, batch, 0)
    _check(got, oracle_batch(batch, 0, scores=DNA_BENCH))


def test_scores_past_int16_rerun_in_int32(built, workloads):
    rng = np.random.default_rng(46)
    big = "".join(rng.choice(list("ACGT"), 12_000))
    batch = workloads.PairBatch.concat([workloads.PairBatch.from_strings(0, [big, big[:11_500]], [big, big[500:]]),
                                        workloads.plain_dna(40, seed=47)])
    exp = oracle_batch(batch, 0, scores=DNA_BENCH)
    over = int(np.count_nonzero(exp[:, 0] > 32767 - 3))
    assert over >= 1
    got, st = _align(built, batch, 0)
    assert st["reruns"] == over, st
    _check(got, exp)
