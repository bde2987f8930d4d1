"""The walk of one pair by a block's warps: rows around its segments' sizes,
paths that end in any of them, guesses that are far off (unrelated, swapped and
overhanging sequences), gaps longer than a warp, free gaps, and records that do
not fit shared memory.  Rows and coordinates equal the oracle's."""
import numpy as np
import pytest

from oracle import oracle as O
from tweakseq_gb300 import aligner as A
from tweakseq_gb300 import workloads as W

pytestmark = pytest.mark.gpu

FIELDS = ("score", "a_begin", "a_end", "b_begin", "b_end", "n_ident", "n_cols")


def dna(rng, n):
    return W.DNA_LETTERS[rng.integers(0, 4, n)]


def partner(rng, a, kind):
    if kind == "related":
        return W._mutate_dna(rng, a, 0.10, 0.02, 3.0)
    if kind == "unrelated":
        return dna(rng, int(rng.integers(1, 2 * len(a) + 2)))
    if kind == "overhang":
        return np.concatenate([dna(rng, int(rng.integers(40, 900))), W._mutate_dna(rng, a, 0.1, 0.02, 40.0), dna(rng, 77)])
    return np.concatenate([a[len(a) // 2:], a[:len(a) // 2]])  # swapped halves


def same(a, b, local, go, ge):
    for output in ("alignment", "identity"):
        got = A.align_pair(a, b, matrix="dna", gap_open=go, gap_extend=ge, mode="local" if local else "global",
                           output=output)
        want = (O.align(a, b, which=O.DNA, gap_open=go, gap_extend=ge, local=local) if output == "alignment" else
                O.score(a, b, which=O.DNA, gap_open=go, gap_extend=ge, local=local, ident=True))
        for f in FIELDS:
            assert getattr(got, f) == getattr(want, f), (f, output, len(a), len(b), local, go, ge)
        if output == "alignment":
            assert (got.aln_a, got.aln_b) == (want.aln_a, want.aln_b), (len(a), len(b), local, go, ge)


@pytest.mark.parametrize("kind", ["related", "unrelated", "overhang", "swapped"])
@pytest.mark.parametrize("local", [False, True])
def test_rows_at_segment_edges(kind, local):
    rng = np.random.default_rng(len(kind))
    for m in (1, 2, 31, 63, 64, 65, 127, 128, 129, 191, 193, 1000, 2047, 2048, 2049, 2300):
        a = dna(rng, m)
        b = partner(rng, a, kind)
        for go, ge in ((5, 2), (0, 0), (0, 1), (30, 0)):
            same(a.tobytes(), b.tobytes(), local, go, ge)
            same(b.tobytes(), a.tobytes(), local, go, ge)


# 32,768 rows and more have room in memory for their records; above 38,400 they
# use it.
@pytest.mark.parametrize("m", [32767, 32768, 38399, 38400, 50001])
@pytest.mark.parametrize("local", [False, True])
def test_records_outside_shared_memory(m, local):
    rng = np.random.default_rng(m)
    a = dna(rng, m)
    b = W._mutate_dna(rng, a[m // 3:m // 3 + 700], 0.1, 0.02, 3.0)
    same(a.tobytes(), b.tobytes(), local, 5, 2)


@pytest.mark.parametrize("local", [False, True])
def test_long_pairs_beside_short_ones(local):
    """One launch walks the long pairs, another the rest of the batch."""
    rng = np.random.default_rng(9)
    seqs = []
    for k in range(400):
        a = dna(rng, int(rng.integers(2500, 4000)) if k % 40 == 7 else int(rng.integers(1, 200)))
        seqs += [a.tobytes(), partner(rng, a, ("related", "overhang")[k % 2]).tobytes()]
    ps = W._pairset_from_lists(seqs, [(2 * k, 2 * k + 1) for k in range(400)], matrix=W.DNA)
    want, sa, sb = O.batch(ps.seqs, ps.a_off, ps.a_len, ps.b_off, ps.b_len, O.DNA, 5, 2, local, O.MODE_ALIGN, 0, True)
    for graph in (False, True):
        got = A.align_batch(ps, matrix="dna", gap_open=5, gap_extend=2, mode="local" if local else "global",
                            use_graph=graph)
        for f in FIELDS:
            assert np.array_equal(got.table[f], want[f]), f
        assert got.aln_a == sa and got.aln_b == sb
