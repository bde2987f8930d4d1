"""GPU tests of the consensus kernel and the guide-tree kernels against the
oracle: bit-exact consensus bytes and per-column figures, identical joins
(ids, positions, distances, heights, branch lengths)."""
import numpy as np
import pytest

from oracle import oracle as O
from tweakseq_gb300 import _native as N
from tweakseq_gb300 import aligner as A
from tweakseq_gb300 import build as B
from tweakseq_gb300 import msa
from tweakseq_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    B.build()
    O.build()


def _family_msa(rng, nseq, ncols, gap=0.15, conserve=0.6):
    """Rows sharing a column profile: each column has a favourite residue
    kept with probability `conserve`, gaps with probability `gap`."""
    fav = W.random_protein(rng, ncols)
    rows = np.empty((nseq, ncols), dtype=np.uint8)
    for k in range(nseq):
        r = W.random_protein(rng, ncols)
        keep = rng.random(ncols) < conserve
        r[keep] = fav[keep]
        r[rng.random(ncols) < gap] = ord("-")
        rows[k] = r
    return rows


def _check_consensus(rows, plurality=None):
    got = msa.consensus(rows, plurality)
    want = O.consensus(rows, -1.0 if plurality is None else plurality)
    assert got.sequence == want[0]
    assert np.array_equal(got.best_score, want[1]) and np.array_equal(got.best_matches, want[2])


@pytest.mark.parametrize("nseq,ncols", [(1, 5), (2, 1), (3, 33), (7, 64), (64, 500), (1000, 97), (3000, 200)])
def test_consensus_matches_oracle(nseq, ncols):
    rng = np.random.default_rng(nseq * 1000 + ncols)
    _check_consensus(_family_msa(rng, nseq, ncols))


def test_consensus_every_byte_class_and_plurality():
    rng = np.random.default_rng(11)
    alphabet = np.frombuffer(b"AAGGLLWWC-.-aJOUXBZ*\x00\x80\xff", dtype=np.uint8)
    for nseq in (2, 5, 40):
        rows = rng.choice(alphabet, size=(nseq, 300)).astype(np.uint8)
        for plur in (None, 0.0, 1.0, nseq / 3.0, float(nseq)):
            _check_consensus(rows, plur)


@pytest.mark.parametrize("first", [0, 31, 32, 33, 64, 99])
def test_consensus_winner_found_past_the_first_rows(first):
    """Gaps down to row `first`, then W: W wins every column and its first
    row is `first` (the warp scans 32 rows per step)."""
    rows = np.full((100, 40), ord("-"), dtype=np.uint8)
    rows[first:, :] = ord("W")
    rows[first:, 7] = ord("C")
    _check_consensus(rows)
    _check_consensus(rows, plurality=5.0)


def test_consensus_device_entry_point():
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(12)
    rows = _family_msa(rng, 500, 300)
    stride = 320
    host = np.zeros((500, stride), dtype=np.uint8)
    host[:, :300] = rows
    d_rows = torch.from_numpy(host).cuda()
    d_out = torch.zeros(300, dtype=torch.uint8, device="cuda")
    d_sc = torch.zeros(300, dtype=torch.int32, device="cuda")
    d_mt = torch.zeros(300, dtype=torch.int32, device="cuda")
    nbytes = N.lib().tsq_consensus_scratch_bytes(300)
    scratch = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream()
    rc = N.lib().tsq_consensus_device(d_rows.data_ptr(), 500, 300, stride, -1.0, d_out.data_ptr(), d_sc.data_ptr(),
                                      d_mt.data_ptr(), scratch.data_ptr(), nbytes, stream.cuda_stream)
    assert rc == 0
    stream.synchronize()
    want = O.consensus(rows)
    assert d_out.cpu().numpy().tobytes() == want[0]
    assert np.array_equal(d_sc.cpu().numpy(), want[1]) and np.array_equal(d_mt.cpu().numpy(), want[2])
    # Too little scratch is refused before anything runs.
    assert N.lib().tsq_consensus_device(d_rows.data_ptr(), 500, 300, stride, -1.0, d_out.data_ptr(), None, None,
                                        scratch.data_ptr(), nbytes - 1, stream.cuda_stream) == N.E_INVALID_ARG


def test_consensus_bad_arguments():
    L = N.lib()
    buf = np.zeros(16, dtype=np.uint8)
    out = np.zeros(16, dtype=np.uint8)
    assert L.tsq_consensus(buf.ctypes.data, 0, 4, 4, -1.0, out.ctypes.data, None, None) == N.E_INVALID_ARG
    assert L.tsq_consensus(buf.ctypes.data, 2, 8, 4, -1.0, out.ctypes.data, None, None) == N.E_INVALID_ARG
    assert L.tsq_consensus(None, 2, 4, 4, -1.0, out.ctypes.data, None, None) == N.E_INVALID_ARG


def _same_tree(tree, want):
    got = tree.nodes
    assert len(got) == len(want)
    for f in N.TREE_NODE_DTYPE.names:
        assert np.array_equal(got[f], want[f]), f


def _tied_identities(rng, n, levels=5):
    """Identities on a coarse grid so that many pairs tie."""
    npairs = n * (n - 1) // 2
    cols = np.full(npairs, 100, dtype=np.int32)
    ident = (rng.integers(0, levels, npairs) * (100 // levels)).astype(np.int32)
    return ident, cols


@pytest.mark.parametrize("method", ["upgma", "nj"])
@pytest.mark.parametrize("n", [2, 3, 17, 200, 600])
def test_tree_matches_oracle(method, n):
    rng = np.random.default_rng(n)
    ident, cols = _tied_identities(rng, n)
    D = O.identity_distances(n, ident, cols)
    want = O.guide_tree(D, N.TREE[method])
    _same_tree(msa.guide_tree(n, ident, cols, method), want)
    _same_tree(msa.guide_tree_from_distances(D, method), want)


@pytest.mark.parametrize("method", ["upgma", "nj"])
def test_tree_from_continuous_identities(method):
    rng = np.random.default_rng(21)
    n = 400
    npairs = n * (n - 1) // 2
    cols = rng.integers(200, 700, npairs).astype(np.int32)
    ident = (cols * rng.uniform(0.1, 0.6, npairs)).astype(np.int32)
    want = O.guide_tree(O.identity_distances(n, ident, cols), N.TREE[method])
    _same_tree(msa.guide_tree(n, ident, cols, method), want)


@pytest.mark.parametrize("method", ["upgma", "nj"])
def test_tree_from_device_resident_all_vs_all(method):
    ps = W.guide_tree_families(n_families=3, per_family=40, seed=41)
    n = 120
    assert len(ps) == n * (n - 1) // 2
    with A.Batch(ps, output="identity") as b:
        b.run()
        tree = msa.guide_tree_from_batch(b, n, method)
        res = b.results()
    want = O.guide_tree(O.identity_distances(n, res.table["n_ident"], res.table["n_cols"]), N.TREE[method])
    _same_tree(tree, want)
    assert sorted(tree.leaf_order()) == list(range(n))
    assert tree.newick().count("(") == n - 1


def test_tree_bad_arguments():
    L = N.lib()
    D = np.array([[0, 1, 2], [1, 0, 3], [2, 4, 0]], dtype=np.int64)  # not symmetric
    out = np.zeros(2, dtype=N.TREE_NODE_DTYPE)
    assert L.tsq_guide_tree_dist(3, D.ctypes.data, 0, out.ctypes.data) == N.E_INVALID_ARG
    assert L.tsq_guide_tree_dist(3, D.ctypes.data, 7, out.ctypes.data) == N.E_INVALID_ARG
    ident = np.array([1, 2, 3], dtype=np.int32)
    cols = np.array([2, 1, 4], dtype=np.int32)  # n_ident > n_cols
    assert L.tsq_guide_tree(3, ident.ctypes.data, cols.ctypes.data, 0, out.ctypes.data) == N.E_INVALID_ARG
    # A batch that is not an all-vs-all, or holds scores only.
    ps = W.guide_tree_families(n_families=1, per_family=5, seed=3)
    with A.Batch(ps, output="identity") as b:
        b.run()
        assert L.tsq_batch_guide_tree(b._h, 4, 0, out.ctypes.data) == N.E_INVALID_ARG
    sub = ps.subset(np.array([1, 0, 2, 3, 4, 5, 6, 7, 8, 9]))
    with A.Batch(sub, output="identity") as b:
        b.run()
        assert L.tsq_batch_guide_tree(b._h, 5, 0, np.zeros(4, dtype=N.TREE_NODE_DTYPE).ctypes.data) == N.E_INVALID_ARG
    with A.Batch(ps, output="score") as b:
        b.run()
        assert L.tsq_batch_guide_tree(b._h, 5, 0, np.zeros(4, dtype=N.TREE_NODE_DTYPE).ctypes.data) == N.E_INVALID_ARG


@pytest.mark.parametrize("method", ["upgma", "nj"])
@pytest.mark.parametrize("kind", ["all equal", "duplicates", "negative", "1100 leaves"])
def test_tree_rows_that_tie_or_never_settle(method, kind):
    """Distances that leave every row open, tie most pairs, or lie below zero;
    more rows to scan than one join keeps results of."""
    rng = np.random.default_rng(83)
    n = 1100 if kind == "1100 leaves" else 130
    if kind == "all equal":
        D = np.full((n, n), 1 << 31, dtype=np.int64)
    elif kind == "duplicates":
        base = np.triu(rng.integers(1 << 30, 1 << 32, (n, n)), 1)
        g = rng.integers(0, n // 3, n)
        D = (base + base.T)[np.ix_(g, g)]
    else:
        lo = -(1 << 31) if kind == "negative" else 0
        base = np.triu(rng.integers(lo, 1 << 32, (n, n)), 1)
        D = base + base.T
    np.fill_diagonal(D, 0)
    D = np.ascontiguousarray(D, dtype=np.int64)
    _same_tree(msa.guide_tree_from_distances(D, method), O.guide_tree(D, N.TREE[method]))


def test_tree_of_more_leaves_than_one_cluster_holds():
    """The first joins by two launches each, the rest in one cluster."""
    n = 3340
    rng = np.random.default_rng(84)
    ident, cols = _tied_identities(rng, n, levels=50)
    want = O.guide_tree(O.identity_distances(n, ident, cols), N.TREE["upgma"])
    _same_tree(msa.guide_tree(n, ident, cols, "upgma"), want)


# Tiles of 128 columns, warps of 32 rows apart in pairs: ragged columns, rows
# without a partner, one tile and many, one slice of rows per tile and 152, the
# even split (110 tiles), and a split that leaves some blocks without rows.
@pytest.mark.parametrize("nseq,ncols", [(6145, 409), (2500, 1003), (701, 5003), (200, 14000),
                                        (31, 130001)])
def test_consensus_pair_counts_at_tile_and_row_edges(nseq, ncols):
    rng = np.random.default_rng(nseq + ncols)
    rows = _family_msa(rng, min(nseq, 500), ncols)[rng.integers(0, min(nseq, 500), nseq)]
    rows[rng.integers(0, nseq, 40), rng.integers(0, ncols, 40)] = rng.integers(0, 256, 40)
    _check_consensus(rows)


def test_consensus_pair_counters_do_not_wrap_and_run_captured():
    """More rows than 16-bit counters hold per block, all alike; then random
    rows through the same captured launches."""
    torch = pytest.importorskip("torch")
    nseq, ncols = 21_000_003, 4
    rows = torch.empty((nseq, ncols), dtype=torch.uint8, device="cuda")
    out = torch.zeros(ncols, dtype=torch.uint8, device="cuda")
    score = torch.zeros(ncols, dtype=torch.int32, device="cuda")
    match = torch.zeros(ncols, dtype=torch.int32, device="cuda")
    nbytes = N.lib().tsq_consensus_scratch_bytes(ncols)
    scratch = torch.empty(nbytes, dtype=torch.uint8, device="cuda")

    def run():
        rc = N.lib().tsq_consensus_device(rows.data_ptr(), nseq, ncols, ncols, -1.0, out.data_ptr(), score.data_ptr(),
                                          match.data_ptr(), scratch.data_ptr(), nbytes,
                                          torch.cuda.current_stream().cuda_stream)
        assert rc == 0

    rows[:] = ord("A")
    rows[:, 2] = ord("-")
    run()
    assert out.cpu().numpy().tobytes() == b"AA-A"
    assert score.tolist() == [4 * (nseq - 1)] * 2 + [nseq - 1] + [4 * (nseq - 1)]
    assert match.tolist() == [nseq - 1] * 4
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run()
    letters = torch.tensor(list(b"ACDW"), dtype=torch.uint8, device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(3)
    rows.copy_(letters[torch.randint(0, 4, (nseq, ncols), device="cuda", generator=gen)])
    graph.replay()
    torch.cuda.synchronize()
    count = torch.stack([(rows == int(x)).sum(0) for x in letters]).cpu().numpy().astype(np.int64)
    # A, C, D, W against A, C, D, W (BLOSUM62); a letter's matches are its own
    # rows, the only positive pairs here.  C's sum is the largest: 0 + 9 - 3 - 2.
    pair = np.array([[4, 0, -2, -3], [0, 9, -3, -2], [-2, -3, 6, -4], [-3, -2, -4, 11]])
    sums = pair @ count - np.diag(pair)[:, None]
    assert (sums.argmax(0) == 1).all()
    assert np.array_equal(score.cpu().numpy(), sums[1]) and np.array_equal(match.cpu().numpy(), count[1] - 1)
    assert out.cpu().numpy().tobytes() == bytes(ord("C") if c - 1 >= nseq / 2 else ord("?") for c in count[1])
