"""wait_polls counts the polls of a wait, however long a strip sleeps between
two of them while its turn is far off."""
import numpy as np
import pytest

from oracle import oracle as O
from tweakseq_gb300 import _native as N
from tweakseq_gb300 import aligner as A
from tweakseq_gb300 import build as B
from tweakseq_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    B.build()
    O.build()


@pytest.mark.parametrize("lane", ["auto", "i32"])
def test_few_polls_are_enough_for_strips_far_from_their_turn(lane):
    """All strips of a lone pair start at once; the last one's turn comes after
    milliseconds, some hundred sleeps."""
    rng = np.random.default_rng(58)
    a = W.DNA_LETTERS[rng.integers(0, 4, 100_000)]
    b = W._mutate_dna(rng, a, 0.1, 0.02, 3.0)[:2000]
    ps = W._pairset_from_lists([a.tobytes(), b.tobytes()], [(0, 1)], matrix=W.DNA)
    kw = dict(matrix="dna", gap_open=5, gap_extend=2, output="score", lane=lane)
    want = O.score(a.tobytes(), b.tobytes(), which=O.DNA, gap_open=5, gap_extend=2)
    for _ in range(3):
        got = A.align_batch(ps, wait_polls=2000, **kw)
        assert got.table["score"][0] == want.score


@pytest.mark.parametrize("lane", ["auto", "i32"])
@pytest.mark.parametrize("polls", [1, 3, 40])
def test_a_pair_whose_waits_run_out_holds_up_no_other(lane, polls):
    """The last strips' turn comes after more sleeps than that: the long pair
    reports it, the others and the next call on the same engine are right."""
    rng = np.random.default_rng(59)
    a = W.DNA_LETTERS[rng.integers(0, 4, 200_000)]
    seqs = [a.tobytes(), a[500:1500].tobytes()]
    for k in range(20):
        x = W.DNA_LETTERS[rng.integers(0, 4, 700 + 90 * (k % 3))]
        seqs += [x.tobytes(), W._mutate_dna(rng, x, 0.1, 0.02, 3.0).tobytes()]
    ps = W._pairset_from_lists(seqs, [(2 * k, 2 * k + 1) for k in range(21)], matrix=W.DNA)
    kw = dict(matrix="dna", gap_open=5, gap_extend=2, output="alignment", mode="local", lane=lane)
    want, sa, sb = O.batch(ps.seqs, ps.a_off, ps.a_len, ps.b_off, ps.b_len, O.DNA, 5, 2, True, O.MODE_ALIGN, 0, True)
    for limit in (polls, 0):
        got = A.align_batch(ps, wait_polls=limit, check=False, **kw)
        assert got.table["status"][0] == (N.E_TIMEOUT if limit else 0)
        ok = got.table["status"] == 0
        # (A short pair's second strip may be short of polls as well.)
        assert ok[1:].all() or limit
        for k in np.flatnonzero(ok):
            assert got.table["score"][k] == want["score"][k]
            assert got.aln_a[k] == sa[k] and got.aln_b[k] == sb[k]
