"""Admission by memory: a request that fits the budget by its residues, records
and boundary rows is taken.  Long pairs' rows take the place of boundary rows
that those pairs do not use; other pairs have none."""
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


def _warps():
    torch = pytest.importorskip("torch")
    return torch.cuda.get_device_properties(0).multi_processor_count * 16


def _budget(ps):
    """Residues and codes, 80 bytes a pair, and eight boundary rows of 16 bytes
    a column for each of the launch's warps."""
    n, warps = len(ps), _warps()
    return 2 * len(ps.seqs) + 256 + 80 * n + min(warps, n + 8) * 8 * (int(ps.b_len.max()) + 64) * 16


def _pairs(rng, n, lo, hi, dna):
    letters = W.DNA_LETTERS if dna else np.frombuffer(b"ARNDCQEGHILKMFPSTWYV", dtype=np.uint8)
    seqs = []
    for _ in range(n):
        a = letters[rng.integers(0, len(letters), int(rng.integers(lo, hi + 1)))]
        b = np.where(rng.random(len(a)) < 0.8, a, letters[rng.integers(0, len(letters), len(a))])
        seqs += [a.tobytes(), b[:max(1, len(a) - int(rng.integers(0, 9)))].astype(np.uint8).tobytes()]
    kw = dict(matrix=W.DNA, gap_open=5, gap_extend=2) if dna else {}
    return W._pairset_from_lists(seqs, [(2 * k, 2 * k + 1) for k in range(n)], **kw)


# Fewer pairs than warps, of which some may be long; more pairs than warps, none
# of which is (at most 600 columns in one strip; an identity request).
@pytest.mark.parametrize("n,lo,hi,dna,output,mode", [
    (2000, 200, 500, False, "score", "global"),
    (60, 4000, 5000, True, "score", "local"),
    (4, 39000, 39100, True, "score", "global"),
    (5000, 50, 250, False, "score", "global"),
    (5000, 200, 400, False, "identity", "global"),
])
def test_request_of_exactly_the_budget_is_taken(n, lo, hi, dna, output, mode):
    ps = _pairs(np.random.default_rng(n + lo), n, lo, hi, dna)
    kw = dict(matrix="dna", gap_open=5, gap_extend=2) if dna else {}
    want = A.align_batch(ps, output=output, mode=mode, **kw)
    budget = _budget(ps)
    with A.Server(slots=2, hbm_budget_bytes=budget) as srv:
        got = srv.poll(srv.submit(ps, output=output, mode=mode, **kw))
        st = srv.stats()
    assert st["rejected"] == 0
    assert st["peak_reserved_bytes"] <= budget
    for f in ("score", "a_end", "b_end", "n_ident", "n_cols", "status"):
        assert np.array_equal(got.table[f], want.table[f]), f
