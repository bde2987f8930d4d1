"""wait_polls counts the polls of a wait, however long a strip sleeps between
two of them while its turn is far off."""
import numpy as np
import pytest

from oracle import oracle as O
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
