"""Strip fills (one pair over many warps) at the sizes where they can go wrong:
strip and lane edges, hand-over chunks, odd column counts, extreme gap costs,
invalid residues in one strip of many.  Every result equals the oracle's."""
import numpy as np
import pytest

from oracle import oracle as O
from tweakseq_gb300 import _native as N
from tweakseq_gb300 import aligner as A
from tweakseq_gb300 import workloads as W

pytestmark = pytest.mark.gpu

FIELDS = ("score", "a_begin", "a_end", "b_begin", "b_end", "n_ident", "n_cols")
# Lanes of four and eight rows, strips of 128 and 512, chunks of 8 and 32
# columns; a length of one.
EDGES = [1, 3, 4, 5, 31, 33, 63, 127, 128, 129, 255, 257, 511, 512, 513]


def related(rng, m, n):
    """A DNA-like pair of exactly m and n residues that share a stretch."""
    a = W.DNA_LETTERS[rng.integers(0, 4, m)]
    b = W.DNA_LETTERS[rng.integers(0, 4, n)]
    k = int(0.7 * min(m, n))
    if k:
        i, j = rng.integers(0, m - k + 1), rng.integers(0, n - k + 1)
        b[j:j + k] = np.where(rng.random(k) < 0.9, a[i:i + k], b[j:j + k])
    return a.tobytes(), b.tobytes()


def want_of(a, b, output, local, go, ge):
    if output == "alignment":
        return O.align(a, b, which=O.DNA, gap_open=go, gap_extend=ge, local=local)
    return O.score(a, b, which=O.DNA, gap_open=go, gap_extend=ge, local=local, ident=output == "identity")


@pytest.mark.parametrize("output", ["score", "identity", "alignment"])
@pytest.mark.parametrize("local", [False, True])
def test_one_pair_at_strip_edges(output, local):
    rng = np.random.default_rng(71)
    mode = "local" if local else "global"
    for m in EDGES:
        for n in rng.choice(EDGES, 5, replace=False).tolist() + [m]:
            a, b = related(rng, m, n)
            # The last: a gap opening beyond the entry's 20 bits of H - F when uncut.
            for go, ge in ((5, 2), (0, 1), (900000, 3)):
                got = A.align_pair(a, b, matrix="dna", gap_open=go, gap_extend=ge, mode=mode, output=output)
                o = want_of(a, b, output, local, go, ge)
                for f in FIELDS:
                    assert getattr(got, f) == getattr(o, f), (f, m, n, go, ge)
                if output == "alignment":
                    assert (got.aln_a, got.aln_b) == (o.aln_a, o.aln_b), (m, n, go, ge)


@pytest.mark.parametrize("output", ["score", "alignment"])
@pytest.mark.parametrize("local", [False, True])
def test_full_gpu_of_long_pairs_at_strip_edges(output, local):
    """Enough pairs to fill every scheduler, so the int16x2 strips run, with
    one- and two-row last strips, short second sequences and a pair whose
    rows are empty."""
    rng = np.random.default_rng(72)
    seqs, pairs = [], []
    sizes = [(513, 901), (514, 1024), (1024, 700), (1025, 769), (1537, 65), (2049, 33), (900, 1801), (0, 700)]
    for k in range(320):
        m, n = sizes[k % len(sizes)]
        seqs += list(related(rng, m, n))
        pairs.append((2 * k, 2 * k + 1))
    ps = W._pairset_from_lists(seqs, pairs, matrix=W.DNA)
    mode = O.MODE_ALIGN if output == "alignment" else O.MODE_SCORE
    want = O.batch(ps.seqs, ps.a_off, ps.a_len, ps.b_off, ps.b_len, O.DNA, 5, 2, local, mode, 0, output == "alignment")
    if output == "alignment":
        want, sa, sb = want
    got = A.align_batch(ps, matrix="dna", gap_open=5, gap_extend=2, mode="local" if local else "global", output=output)
    for f in FIELDS if output == "alignment" else ("score", "a_end", "b_end"):
        assert np.array_equal(got.table[f], want[f]), f
    if output == "alignment":
        assert got.aln_a == sa and got.aln_b == sb


@pytest.mark.parametrize("where", ["first strip", "last strip", "b"])
def test_invalid_residue_in_one_strip(where):
    rng = np.random.default_rng(73)
    a, b = related(rng, 700, 650)
    x, y = bytearray(a), bytearray(b)
    if where == "b":
        y[640] = ord("!")
    else:
        x[5 if where == "first strip" else 699] = ord("!")
    for output in ("score", "identity", "alignment"):
        with pytest.raises(N.TsqError) as e:
            A.align_pair(bytes(x), bytes(y), matrix="dna", gap_open=5, gap_extend=2, output=output)
        assert e.value.rc == N.E_INVALID_RESIDUE
    # The cached path is usable afterwards.
    assert A.align_pair(a, b, matrix="dna", gap_open=5, gap_extend=2, output="score").score == \
        O.score(a, b, which=O.DNA, gap_open=5, gap_extend=2).score


@pytest.mark.parametrize("local", [False, True])
@pytest.mark.parametrize("lane", ["auto", "i16", "i32"])
def test_identity_from_planes_equals_carried_counts(monkeypatch, local, lane):
    """Identity output walks traceback planes where they fit in memory and
    carries the counts through the fill where they do not: the same table
    either way (an empty pair and an invalid residue among them), and the
    oracle's on a sample."""
    ps = W.uneven_pairs(n_pairs=1500, seed=74)
    seqs, tab = A._as_inputs(ps)
    seqs, tab = seqs.copy(), tab.copy()
    tab["a_len"][7] = 0
    seqs[int(tab["b_off"][9]) + 2] = ord("?")
    pairs = (seqs, tab["a_off"], tab["a_len"], tab["b_off"], tab["b_len"])
    kw = dict(output="identity", mode="local" if local else "global", lane=lane, check=False)
    got = A.align_batch(pairs, **kw)
    monkeypatch.setenv("TSQ_WAVE_BUDGET_BYTES", "1")
    want = A.align_batch(pairs, **kw)
    assert got.table["status"][9] == want.table["status"][9] == N.E_INVALID_RESIDUE
    ok = np.arange(1500) != 9
    for f in FIELDS + ("status",):
        assert np.array_equal(got.table[f][ok], want.table[f][ok]), f
    idx = np.arange(20, 1500, 31)
    o = O.batch(seqs, tab["a_off"][idx], tab["a_len"][idx], tab["b_off"][idx], tab["b_len"][idx], O.BLOSUM62, 11, 1,
                local, O.MODE_IDENT)
    for f in ("score", "n_ident", "n_cols"):
        assert np.array_equal(got.table[f][idx], o[f]), f
