"""Large calls in chunks whose residues go up in segments: pairs that share
sequences, so that the first chunk already reads to the end of the buffer, whose
length is no multiple of the segments' grain."""
import numpy as np
import pytest

from oracle import oracle as O
from tweakseq_gb300 import aligner as A
from tweakseq_gb300 import build as B

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    B.build()
    O.build()


@pytest.mark.parametrize("tail", [0, 1, 4, 15])
@pytest.mark.parametrize("output", ["score", "identity"])
def test_all_vs_all_of_shared_sequences(output, tail):
    n = 260  # 33,670 pairs
    rng = np.random.default_rng(tail)
    lens = rng.integers(5, 60, n)
    lens[-1] += (tail - int(lens.sum())) % 16
    assert lens.sum() % 16 == tail
    off = np.concatenate([[0], np.cumsum(lens)[:-1]])
    seqs = np.frombuffer(b"ARNDCQEGHILKMFPSTWYV", dtype=np.uint8)[rng.integers(0, 20, int(lens.sum()))]
    i, j = np.triu_indices(n, 1)
    got = A.align_batch((seqs, off[i], lens[i], off[j], lens[j]), output=output).table
    mode = O.MODE_IDENT if output == "identity" else O.MODE_SCORE
    want = O.batch(seqs, off[i], lens[i], off[j], lens[j], O.BLOSUM62, 11, 1, False, mode)
    for f in ("score", "n_ident", "n_cols") if output == "identity" else ("score",):
        assert np.array_equal(got[f], want[f]), f
