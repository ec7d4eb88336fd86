"""CPU check of the reverse band's lower side (reverse_low_band / band_last_row in
gpu-bsw_gb300/csrc/sw_common.cuh).

Every cell (r, c) of an alignment reaching the forward score satisfies
r <= c + (match * rows - score) // match, so a strip of columns ends at its last
column's row bound (rounded up to even), and the next strip reads the zero state
past it.  The strip layout of the kernels, cut on both sides, finds the same
first cell reaching the score as the full DP.
"""
import importlib

import numpy as np
import pytest

import oracle
from test_reverse_band import _band, _band_first_row, _penalty

wl = importlib.import_module("gpu-bsw_gb300.workloads")


def _band_last_row(last_col, low, nrows):
    r = last_col + low
    return min(r + (r & 1), nrows)


def _first_hit(L, S, scores, target, band, low, W):
    match, mismatch, open_, ext = scores
    n, m = len(S), len(L)
    nstrips = -(-min(m, n + band) // W)
    width = nstrips * W
    first = [_band_first_row(s * W + 1, band) for s in range(nstrips)]
    last = [_band_last_row(s * W + W, low, n) for s in range(nstrips)]
    H = np.zeros((n + 1, width + 1), np.int64)
    E = np.zeros((n + 1, width + 1), np.int64)
    F = np.zeros((n + 1, width + 1), np.int64)
    computed = 0
    for r in range(1, n + 1):
        for c in range(1, width + 1):
            s = (c - 1) // W
            if r < first[s] or r > last[s]:
                continue  # not computed: the zero state
            computed += 1
            E[r, c] = max(0, E[r, c - 1] + ext, H[r, c - 1] + open_)
            F[r, c] = max(0, F[r - 1, c] + ext, H[r - 1, c] + open_)
            score = (match if S[r - 1] == L[c - 1] else mismatch) if c <= m else -128
            H[r, c] = max(0, H[r - 1, c - 1] + score, E[r, c], F[r, c])
        hits = np.nonzero(H[r, 1:] == target)[0]
        if len(hits):
            return (r, int(hits[0]) + 1), computed
    return None, computed


@pytest.mark.parametrize("W", [4, 16, 64])
@pytest.mark.parametrize("scores", [(3, -3, -6, -1), (1, -3, -3, -1), (5, -4, -8, -2)])
def test_strips_cut_on_both_sides_find_the_begin(scores, W):
    batch = wl.custom_dna(60, 21 + scores[0], 20, 90, 10, 70, related=0.8)
    p = _penalty(scores)
    res = oracle.align(oracle.DNA, batch.ref, batch.ref_off, batch.query, batch.query_off, scores=scores)
    cut = 0
    for k in range(batch.n):
        s, rb, re_, qb, qe = (int(v) for v in res[k])
        ref, qry = batch.strings(k)
        if s <= 0 or (band := _band(len(ref), len(qry), re_, qe, s, scores[0], p)) < 0:
            continue
        A, B = ref[:re_][::-1], qry[:qe][::-1]
        L, S = (A, B) if re_ >= qe else (B, A)
        low = (scores[0] * len(S) - s) // scores[0]
        begin = (qe - qb, re_ - rb) if re_ >= qe else (re_ - rb, qe - qb)
        hit, computed = _first_hit(L, S, scores, s, band, low, W)
        assert hit == begin, (k, s, band, low)
        cut += computed < _first_hit(L, S, scores, s, band, len(S), W)[1]
    assert W == 64 or cut > 5
