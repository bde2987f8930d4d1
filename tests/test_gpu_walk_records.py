"""One pair whose walk keeps its records in global memory, in front of the
traceback planes: first sequences of a multiple of 64 rows, and paths through the
planes' first cells, which the last row's record must not reach.  Rows and counts
equal the oracle's."""
import numpy as np
import pytest

from oracle import oracle as O
from tweakseq_gb300 import aligner as A
from tweakseq_gb300 import build as B
from tweakseq_gb300 import workloads as W

pytestmark = pytest.mark.gpu

FIELDS = ("score", "a_begin", "a_end", "b_begin", "b_end", "n_ident", "n_cols")


@pytest.fixture(scope="module", autouse=True)
def built():
    B.build()
    O.build()


def dna(rng, n):
    return W.DNA_LETTERS[rng.integers(0, 4, n)]


def same(a, b, local, outputs=("alignment", "identity")):
    a, b = a.tobytes(), b.tobytes()
    want = O.align(a, b, which=O.DNA, gap_open=5, gap_extend=2, local=local)
    for output in outputs:
        for lane in ("auto", "i32"):
            got = A.align_pair(a, b, matrix="dna", gap_open=5, gap_extend=2, mode="local" if local else "global",
                               output=output, lane=lane)
            fields = FIELDS if output == "alignment" or not local else ("score", "a_end", "b_end", "n_ident", "n_cols")
            for f in fields:
                assert getattr(got, f) == getattr(want, f), (f, output, lane, len(a), len(b), local)
            if output == "alignment":
                assert (got.aln_a, got.aln_b) == (want.aln_a, want.aln_b), (lane, len(a), len(b), local)


@pytest.mark.parametrize("m", [38400, 38464, 40000, 51200])
@pytest.mark.parametrize("local", [False, True])
def test_path_through_the_first_cells(m, local):
    rng = np.random.default_rng(m)
    a = dna(rng, m)
    for n in range(297, 304):
        # b from a's start; from both ends (the local path ends in row m too
        # where the last part is the longer one).
        same(a, a[:n], local)
        same(a, np.concatenate([a[:n // 4], a[m - (n - n // 4):]]), local)


@pytest.mark.parametrize("n", [19199, 19200, 19201])
def test_second_sequence_of_about_half_the_rows(n):
    rng = np.random.default_rng(n)
    a = dna(rng, 38400)
    same(a, W._mutate_dna(rng, a, 0.1, 0.02, 3.0)[:n], False)
