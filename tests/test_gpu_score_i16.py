"""The int16x2 score fill at the sizes where it can go wrong: columns around
the four-step units that row maxima are taken over, ties in later columns and
rows, lane and band edges, scores on both sides of the tagged form's limit, and
gap costs for which the scores do not fit the biased profile bytes.  Every
score and end equals the oracle's."""
import numpy as np
import pytest

from oracle import oracle as O
from tweakseq_gb300 import aligner as A
from tweakseq_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def check(seqs, matrix, which, go, ge, local):
    ps = W._pairset_from_lists(seqs, [(2 * k, 2 * k + 1) for k in range(len(seqs) // 2)], matrix=matrix)
    got = A.align_batch(ps, matrix=which, gap_open=go, gap_extend=ge, mode="local" if local else "global",
                        output="score").table
    want = O.batch(ps.seqs, ps.a_off, ps.a_len, ps.b_off, ps.b_len, matrix, go, ge, local, O.MODE_SCORE)
    for f in ("score", "a_end", "b_end"):
        bad = np.flatnonzero(got[f] != want[f])
        assert not len(bad), (f, go, ge, ps.pair(int(bad[0])))


# The profile bytes hold score + open + ext from 0 to 127 (BLOSUM62: -4 .. 11):
# inside, at both ends, and outside on either side.
@pytest.mark.parametrize("go,ge", [(11, 1), (3, 1), (115, 1), (0, 1), (2, 1), (116, 1), (500, 9)])
@pytest.mark.parametrize("local", [False, True])
def test_lane_band_and_unit_edges(go, ge, local):
    rng = np.random.default_rng(go * 10 + ge)
    ms = [1, 2, 7, 8, 9, 31, 32, 33, 63, 64, 65, 127, 129, 256, 257, 511, 513]
    ns = [1, 2, 3, 4, 5, 6, 7, 8, 9, 15, 16, 17, 31, 63, 64, 65, 66, 67, 130, 258]
    seqs = []
    for m in ms:
        for n in ns:
            a, b = W.random_protein(rng, m), W.random_protein(rng, n)
            k = min(m, n) // 2
            b[:k] = a[:k]
            seqs += [a.tobytes(), b.tobytes()]
            # Equal maxima in every phase of a unit and in several rows.
            p = int(rng.integers(1, 6))
            seqs += [(b"W" + b"P" * p) * (m // (p + 1)) + b"W", b"G" * int(rng.integers(0, 5)) + (b"W" + b"G" * p) * n]
    check(seqs, O.BLOSUM62, "blosum62", go, ge, local)


@pytest.mark.parametrize("local", [False, True])
def test_scores_at_the_tagged_and_checked_limits(local):
    """W against W scores 11: 16,000 is crossed at 1,455 rows, 32,767 at 2,979."""
    rng = np.random.default_rng(5)
    seqs = []
    for m in (1440, 1452, 1453, 1454, 1455, 1500, 2970, 2978, 2979, 2985):
        for n in (m, m + 3, 40):
            b = np.frombuffer(b"W" * n, np.uint8).copy()
            b[rng.integers(0, n, 3)] = ord("A")
            seqs += [b"W" * m, b.tobytes(), b.tobytes(), b"W" * m]
    check(seqs, O.BLOSUM62, "blosum62", 11, 1, local)
