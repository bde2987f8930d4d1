"""Rows that share memory: results released one by one, in any order and on
any thread, leave the others' rows as they were."""
import ctypes
import threading

import numpy as np
import pytest

from oracle import oracle as O
from tweakseq_gb300 import _native as N
from tweakseq_gb300 import aligner as A
from tweakseq_gb300 import workloads as W

pytestmark = pytest.mark.gpu


# One pair, a serial collect, a parallel one whose slices fill several blocks,
# and rows longer than a block.
@pytest.mark.parametrize("pairs,length", [(1, 90), (40, 90), (3000, 300), (6, 150_000)])
def test_results_released_in_any_order(pairs, length):
    rng = np.random.default_rng(pairs)
    seqs = []
    for _ in range(pairs):
        a = W.DNA_LETTERS[rng.integers(0, 4, length)]
        seqs += [a.tobytes(), a[:max(1, length - int(rng.integers(0, 9)))].tobytes()]
    if pairs > 1:
        seqs[3] = b"AC!T"  # this pair has no rows
    if length > 1000:  # long rows from few columns
        seqs = [s if k % 2 == 0 else s[:20] for k, s in enumerate(seqs)]
    ps = W._pairset_from_lists(seqs, [(2 * k, 2 * k + 1) for k in range(pairs)], matrix=W.DNA)
    tab = A.pair_table(ps.a_off, ps.a_len, ps.b_off, ps.b_len)
    p, keep = N.make_params("dna", 5, 2, "global", "alignment", "auto", None)
    raw = np.zeros(pairs, dtype=N.RESULT_DTYPE)
    L = N.lib()
    rc = L.tsq_align_batch(ps.seqs.ctypes.data, len(ps.seqs), tab.ctypes.data, pairs, ctypes.byref(p),
                           ctypes.byref(A._opts()), raw.ctypes.data)
    assert rc == (N.E_INVALID_RESIDUE if pairs > 1 else 0)

    def rows(k):
        r = raw[k]
        return (ctypes.string_at(int(r["aln_a"])), ctypes.string_at(int(r["aln_b"]))) if r["aln_a"] else None

    want = [rows(k) for k in range(pairs)]
    assert [w is None for w in want] == [pairs > 1 and k == 1 for k in range(pairs)]
    for k in (0, pairs // 2, pairs - 1):
        if want[k] is not None:
            o = O.align(seqs[2 * k], seqs[2 * k + 1], which=O.DNA, gap_open=5, gap_extend=2, local=False)
            assert tuple(x.decode() if isinstance(x, bytes) else x for x in want[k]) == (o.aln_a, o.aln_b)
    order = rng.permutation(pairs)
    first, second = order[:pairs // 3], order[pairs // 3:2 * pairs // 3]

    def free(ks):
        for k in ks:
            L.tsq_result_free(raw.ctypes.data + int(k) * raw.itemsize)

    threads = [threading.Thread(target=free, args=(ks,)) for ks in (first, second)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not raw["aln_a"][order[:2 * pairs // 3]].any()
    assert all(rows(k) == want[k] for k in order[2 * pairs // 3:])
    L.tsq_results_free(raw.ctypes.data, pairs)
    assert not raw["aln_a"].any() and not raw["aln_b"].any()
    del keep
