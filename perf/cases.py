"""Performance cases: what a user of the library has it do, by use.

Each case goes through a public entry point (``aligner.align_pair``,
``aligner.align_batch``, ``aligner.Batch``, ``aligner.Server``,
``msa.guide_tree``, ``msa.guide_tree_from_batch``, ``tsq_consensus_device``)
on seeded inputs of the shapes the workloads module describes.  ``listed``
names the cases, ``draw`` gives more of the same ranges, ``prepare`` makes the
inputs, ``run`` is one pass, ``work`` is what a pass cannot do without, and
``exact`` is the same result by plain numpy or torch where that is quick.

All outputs are whole numbers or bytes: scores, coordinates, counts, gapped
rows, tree joins, consensus bytes.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from tweakseq_gb300 import _native as N
from tweakseq_gb300 import aligner as A
from tweakseq_gb300 import msa
from tweakseq_gb300 import workloads as W

# Integer operations of one cell of the three-matrix recurrence: E and F are
# two additions and a maximum each, H one addition and two maxima.
OPS_PER_CELL = 9.0
# Cells of the largest listed case (long_dna); a drawn case stays below it.
MOST_CELLS = 2.5e10

SIGMA = 0.5  # log-normal spread of the protein lengths (as workloads.uneven_pairs)
FIELDS = ("score", "a_begin", "a_end", "b_begin", "b_end", "n_ident", "n_cols", "status")


def listed():
    return [
        # "Align selection" of two sequences in an editor: the smallest call,
        # where the latency of one launch sequence is all there is.
        dict(name="pair_protein", kind="pair", alphabet="protein", length=383, mode="global", output="alignment",
             gap_open=11, gap_extend=1),
        # The same call on a gene-sized DNA pair, local: one pair's own work
        # on an otherwise idle GPU.
        dict(name="pair_dna_local", kind="pair", alphabet="dna", length=3001, mode="local", output="alignment",
             gap_open=5, gap_extend=2),
        # A 20 kb DNA pair, global, with its rows: the plain call's largest.
        dict(name="pair_dna_long", kind="pair", alphabet="dna", length=20011, mode="global", output="alignment",
             gap_open=5, gap_extend=2),
        # All-vs-all of an editor's selection (64 proteins, 2,016 pairs), host
        # buffers in, gapped rows out.
        dict(name="selection_rows", kind="selection", n_seqs=64, lo=200, hi=400, mode="global", output="alignment",
             gap_open=11, gap_extend=1),
        # Uneven protein pairs, score only, host buffers in and results out:
        # the batched call.
        dict(name="uneven_score", kind="batch", alphabet="protein", pairs=40013, median=350, mode="global",
             output="score", gap_open=11, gap_extend=1),
        # One query family against a database, local scores with end
        # coordinates (what a search does before it aligns its hits).
        dict(name="search_local", kind="batch", alphabet="protein", pairs=20011, median=330, mode="local",
             output="score", gap_open=11, gap_extend=1),
        # A device-resident batch of medium size with traceback, run again and
        # read back (realigning a project's pairs).
        dict(name="resident_rows", kind="resident", alphabet="protein", pairs=3001, median=350, mode="global",
             output="alignment", gap_open=10, gap_extend=2),
        # Long DNA pairs (10 to 50 kb) with traceback.
        dict(name="long_dna", kind="long", pairs=23, lo=10000, hi=50000, gap_open=5, gap_extend=2),
        # The first stage of a multiple alignment: identities of all pairs of a
        # few hundred proteins in families, then the UPGMA guide tree, all on
        # the device.
        dict(name="families_upgma", kind="families", families=6, per_family=83, lo=250, hi=600, method="upgma"),
        # A neighbour-joining tree from the identities a program has in hand.
        dict(name="tree_nj", kind="tree", leaves=2003, method="nj"),
        # The consensus line of a large alignment that is on the device.
        dict(name="consensus_large", kind="consensus", rows=100003, cols=2000),
        # A server's mixed requests: 1 to 200 pairs each, protein or DNA, 50
        # to 5,000 residues, traceback on half.
        dict(name="served_mix", kind="served", requests=24, max_pairs=200, lo=50, hi=5000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _gaps(rng, alphabet):
    return rng.choice([(11, 1), (10, 2), (12, 2), (9, 1)] if alphabet == "protein" else [(5, 2), (8, 1), (6, 3)])


def draw(rng):
    kind = rng.choice(["pair", "pair", "selection", "batch", "batch", "resident", "long", "families", "tree",
                       "consensus", "served"])
    if kind == "pair":
        alphabet = rng.choice(["protein", "dna"])
        go, ge = _gaps(rng, alphabet)
        return dict(kind=kind, alphabet=alphabet, length=_log(rng, 20, 5000 if alphabet == "protein" else 24000),
                    mode=rng.choice(["global", "local"]), output=rng.choice(["score", "identity", "alignment"]),
                    gap_open=go, gap_extend=ge)
    if kind == "selection":
        go, ge = _gaps(rng, "protein")
        lo = _log(rng, 50, 400)
        return dict(kind=kind, n_seqs=_log(rng, 4, 80), lo=lo, hi=int(lo * rng.uniform(1.2, 2.5)),
                    mode=rng.choice(["global", "local"]), output=rng.choice(["identity", "alignment"]), gap_open=go,
                    gap_extend=ge)
    if kind in ("batch", "resident"):
        alphabet = rng.choice(["protein", "protein", "dna"])
        go, ge = _gaps(rng, alphabet)
        output = rng.choice(["score", "identity"] if kind == "batch" else ["score", "identity", "alignment"])
        median = _log(rng, 80, 1000)
        most = 4000 if output == "alignment" else 70000
        most = int(min(most, MOST_CELLS / 2 / _mean_square(median)))
        return dict(kind=kind, alphabet=alphabet, pairs=_log(rng, 50, most), median=median,
                    mode=rng.choice(["global", "global", "local"]), output=output, gap_open=go, gap_extend=ge)
    if kind == "long":
        go, ge = _gaps(rng, "dna")
        lo = _log(rng, 6000, 20000)
        return dict(kind=kind, pairs=_log(rng, 2, 24), lo=lo, hi=int(min(50000, lo * rng.uniform(1.1, 3.0))), gap_open=go,
                    gap_extend=ge)
    if kind == "families":
        return dict(kind=kind, families=rng.randint(2, 8), per_family=_log(rng, 8, 60), lo=_log(rng, 100, 300), hi=600,
                    method=rng.choice(["upgma", "nj"]))
    if kind == "tree":
        return dict(kind=kind, leaves=_log(rng, 50, 2200), method=rng.choice(["upgma", "nj"]))
    if kind == "consensus":
        cols = _log(rng, 60, 6000)
        return dict(kind=kind, rows=_log(rng, 20, min(200000, 200_000_000 // cols)), cols=cols)
    return dict(kind="served", requests=rng.randint(4, 32), max_pairs=_log(rng, 8, 200), lo=50,
                hi=_log(rng, 600, 5000))


def _matrix(alphabet):
    return "blosum62" if alphabet == "protein" else "dna"


def _pair_set(case, seed):
    """Uneven pairs of one alphabet (a PairSet)."""
    if case["alphabet"] == "protein":
        return W.uneven_pairs(n_pairs=case["pairs"], median=float(case["median"]), sigma=SIGMA, lo=20,
                              hi=8 * case["median"], seed=seed)
    # DNA pairs of the same lengths: the second sequence with 10 % substitutions
    # and 5 % indels of the first.
    ps = W.uneven_pairs(n_pairs=case["pairs"], median=float(case["median"]), sigma=SIGMA, lo=20,
                        hi=8 * case["median"], ident_lo=0.80, ident_hi=0.95, seed=seed)
    to_dna = np.zeros(256, dtype=np.uint8)
    to_dna[W.AA_LETTERS] = W.DNA_LETTERS[np.arange(20) % 4]
    ps.seqs = to_dna[ps.seqs]
    return ps


def _one_pair(case, seed):
    rng = np.random.default_rng(seed)
    n = case["length"]
    if case["alphabet"] == "protein":
        a = W.random_protein(rng, n)
        sub = (1.0 - rng.uniform(0.30, 0.90)) / (1.0 - float(np.sum(W.AA_FREQ ** 2)))
        b, _ = W._mutate_proteins(rng, a, np.array([n]), np.array([sub]), 0.05)
    else:
        a = W.DNA_LETTERS[rng.integers(0, 4, size=n)]
        b = W._mutate_dna(rng, a, 0.10, 0.02, 3.0)
    if len(b) == 0:
        b = a[:1]
    return a.tobytes(), b.tobytes()


def _params(case, matrix):
    return dict(matrix=matrix, gap_open=case["gap_open"], gap_extend=case["gap_extend"],
                mode=case.get("mode", "global"), output=case.get("output", "alignment"))


def _identities(case, seed):
    """Identical and total columns of the pairs of `leaves` sequences in
    families: 20 to 60 % identity inside one, 4 to 12 % between."""
    rng = np.random.default_rng(seed)
    n = case["leaves"]
    family = rng.integers(0, max(2, n // 100), size=n)
    length = rng.integers(250, 601, size=n)
    depth = rng.uniform(0.20, 0.60, size=n)  # a leaf's own closeness to its family
    i, j = np.triu_indices(n, 1)
    cols = (np.maximum(length[i], length[j]) * rng.uniform(1.0, 1.15, size=len(i))).astype(np.int32)
    share = np.where(family[i] == family[j], np.minimum(depth[i], depth[j]) * rng.uniform(0.9, 1.0, size=len(i)),
                     rng.uniform(0.04, 0.12, size=len(i)))
    return (share * cols).astype(np.int32), cols


def _alignment_rows(case, seed):
    """Rows of a family's alignment: per column one common letter, kept with a
    column's own probability, gaps in some columns (made on the device)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    rows, cols = case["rows"], case["cols"]
    letters = torch.from_numpy(W.AA_LETTERS.copy()).cuda()
    common = letters[torch.randint(0, 20, (cols,), generator=g, device="cuda")]
    kept = torch.rand((cols,), generator=g, device="cuda") * 0.8 + 0.1
    gap = torch.rand((cols,), generator=g, device="cuda") ** 3 * 0.9
    out = torch.empty((rows, cols), dtype=torch.uint8, device="cuda")
    step = max(1, 16_000_000 // cols)
    for r in range(0, rows, step):
        k = min(step, rows - r)
        u = torch.rand((k, cols), generator=g, device="cuda")
        x = letters[torch.randint(0, 20, (k, cols), generator=g, device="cuda")]
        x = torch.where(u < kept, common, x)
        u = torch.rand((k, cols), generator=g, device="cuda")
        out[r:r + k] = torch.where(u < gap, torch.full_like(x, ord("-")), x)
    return out


def _requests(case, seed):
    """A server's traffic: the number of requests, their kinds, sizes and
    lengths are the case's own (as workloads.serving_stream draws them), the
    residues are the seed's."""
    shape, rng = np.random.default_rng(case["requests"]), np.random.default_rng(seed)
    out = []
    for _ in range(case["requests"]):
        pairs = int(np.clip(np.rint(np.exp(shape.uniform(0, np.log(case["max_pairs"])))), 1, case["max_pairs"]))
        dna, rows = bool(shape.random() < 0.5), bool(shape.random() < 0.5)
        seqs = []
        for n in np.rint(np.exp(shape.uniform(np.log(case["lo"]), np.log(case["hi"]), size=pairs))).astype(int):
            if dna:
                a = W.DNA_LETTERS[rng.integers(0, 4, size=n)]
                b = W._mutate_dna(rng, a, 0.10, 0.02, 3.0)
            else:
                a = W.random_protein(rng, n)
                b, _ = W._mutate_proteins(rng, a, np.array([n]), np.array([0.5]), 0.05)
            seqs += [a.tobytes(), b.tobytes() if len(b) else a[:1].tobytes()]
        ps = W._pairset_from_lists(seqs, np.arange(2 * pairs).reshape(-1, 2))
        out.append((ps, dict(matrix="dna" if dna else "blosum62", gap_open=5 if dna else 11, gap_extend=2 if dna else 1,
                             output="alignment" if rows else "score")))
    return out


def _rows_room(case):
    """Bytes that hold the gapped rows of a pass for any seed (each pair's
    two rows have at most as many columns as it has residues)."""
    kind = case["kind"]
    if case.get("output", "alignment") != "alignment" or kind in ("families", "tree", "consensus"):
        return 0
    if kind == "pair":
        residues = 2.3 * case["length"] + 100
    elif kind == "selection":
        residues = case["n_seqs"] * (case["n_seqs"] - 1) * case["hi"]
    elif kind == "long":
        residues = 2.2 * case["pairs"] * case["hi"]
    elif kind == "served":
        residues = 2.2 * case["requests"] * case["max_pairs"] * case["hi"]
    else:
        residues = 3.0 * case["pairs"] * case["median"] + 100 * case["median"]
    return int(2 * residues)


def prepare(case, seed):
    state = _prepare(case, seed)
    state["room"] = _rows_room(case)
    return state


def _prepare(case, seed):
    kind = case["kind"]
    if kind == "pair":
        a, b = _one_pair(case, seed)
        return dict(kind=kind, a=a, b=b, params=_params(case, _matrix(case["alphabet"])))
    if kind == "selection":
        ps = W.all_vs_all_proteins(case["n_seqs"], case["lo"], case["hi"], seed=seed)
        return dict(kind="batch", pairs=ps, params=_params(case, "blosum62"))
    if kind == "batch":
        return dict(kind=kind, pairs=_pair_set(case, seed), params=_params(case, _matrix(case["alphabet"])))
    if kind == "resident":
        ps = _pair_set(case, seed)
        return dict(kind=kind, batch=A.Batch(ps, **_params(case, _matrix(case["alphabet"]))))
    if kind == "long":
        ps = W.long_dna_pairs(case["pairs"], case["lo"], case["hi"], seed=seed)
        return dict(kind="batch", pairs=ps, params=_params(case, "dna"))
    if kind == "families":
        ps = W.guide_tree_families(case["families"], case["per_family"], case["lo"], case["hi"], seed=seed)
        return dict(kind=kind, batch=A.Batch(ps, output="identity"), n=ps.meta["n_seqs"], method=case["method"])
    if kind == "tree":
        ident, cols = _identities(case, seed)
        return dict(kind=kind, n=case["leaves"], ident=ident, cols=cols, method=case["method"])
    if kind == "consensus":
        d = _alignment_rows(case, seed)
        cols = case["cols"]
        bytes_ = N.lib().tsq_consensus_scratch_bytes(cols)
        return dict(kind=kind, rows=d, line=torch.zeros(cols, dtype=torch.uint8, device="cuda"),
                    score=torch.zeros(cols, dtype=torch.int32, device="cuda"),
                    matches=torch.zeros(cols, dtype=torch.int32, device="cuda"),
                    scratch=torch.zeros(bytes_, dtype=torch.uint8, device="cuda"))
    return dict(kind="served", server=A.Server(), requests=_requests(case, seed))


def _in_room(rows, room):
    """Gapped rows back to back, at the head of a buffer of the case's size."""
    out = np.zeros(room, dtype=np.uint8)
    text = "".join(rows).encode("ascii")
    out[:len(text)] = np.frombuffer(text, dtype=np.uint8)
    return out


def _columns(results, room):
    """A list of BatchResult as plain arrays: the table's columns and, where
    there are rows, the gapped rows back to back."""
    out = {f: np.concatenate([r.table[f] for r in results]) for f in FIELDS}
    if room:
        out["rows"] = _in_room([s for r in results if r.aln_a is not None for pair in zip(r.aln_a, r.aln_b) for s in pair],
                               room)
    return out


def _tree(tree):
    return {f: tree.nodes[f] for f in tree.nodes.dtype.names}


def run(state):
    kind = state["kind"]
    if kind == "pair":
        r = A.align_pair(state["a"], state["b"], **state["params"])
        out = {f: getattr(r, f) for f in FIELDS}
        if state["room"]:
            out["rows"] = _in_room([r.aln_a, r.aln_b], state["room"])
        return out
    if kind == "batch":
        return _columns([A.align_batch(state["pairs"], **state["params"])], state["room"])
    if kind == "resident":
        state["batch"].run()
        return _columns([state["batch"].results()], state["room"])
    if kind == "families":
        state["batch"].run()
        tree = msa.guide_tree_from_batch(state["batch"], state["n"], state["method"])
        return {"identities": _columns([state["batch"].results()], state["room"]), "tree": _tree(tree)}
    if kind == "tree":
        return _tree(msa.guide_tree(state["n"], state["ident"], state["cols"], state["method"]))
    if kind == "consensus":
        d = state["rows"]
        N.check(N.lib().tsq_consensus_device(d.data_ptr(), d.shape[0], d.shape[1], d.shape[1], -1.0,
                                             state["line"].data_ptr(), state["score"].data_ptr(),
                                             state["matches"].data_ptr(), state["scratch"].data_ptr(),
                                             state["scratch"].numel(), torch.cuda.current_stream().cuda_stream),
                "tsq_consensus_device")
        return [state["line"], state["score"], state["matches"]]
    ids = [state["server"].submit(ps, **params) for ps, params in state["requests"]]
    return _columns([state["server"].poll(k) for k in ids], state["room"])


def _mean_square(median):
    """Mean of a pair's cells for log-normal lengths of this median."""
    return float(median) ** 2 * math.exp(2 * SIGMA ** 2)


def work(case):
    """Bytes (inputs and results once) and integer operations of one pass, at
    the mean of the case's distribution of lengths."""
    kind = case["kind"]
    if kind == "tree":
        n = case["leaves"]
        pairs = n * (n - 1) // 2
        # Each join writes the joined cluster's distances and finds the next
        # pair among those that are left (one criterion per leaf, at least).
        return {"bytes": 8.0 * pairs + 56.0 * n, "flops": 4.0 * n * n}
    if kind == "consensus":
        rows, cols = case["rows"], case["cols"]
        return {"bytes": rows * cols + 9.0 * cols, "flops": float(rows) * cols}
    if kind == "pair":
        n = case["length"]
        pairs, cells, res = 1, float(n) * n, 2.0 * n
    elif kind == "selection":
        mean = 0.5 * (case["lo"] + case["hi"])
        pairs = case["n_seqs"] * (case["n_seqs"] - 1) // 2
        cells, res = pairs * mean * mean, case["n_seqs"] * mean
    elif kind == "long":
        lo, hi = case["lo"], case["hi"]
        pairs = case["pairs"]
        cells, res = pairs * (hi ** 3 - lo ** 3) / (3.0 * max(1, hi - lo)), pairs * float(lo + hi)
    elif kind == "families":
        n = case["families"] * case["per_family"]
        mean = 0.5 * (case["lo"] + case["hi"])
        pairs = n * (n - 1) // 2
        cells, res = pairs * mean * mean, n * mean
    elif kind == "served":
        lo, hi, k = case["lo"], case["hi"], case["max_pairs"]
        pairs = case["requests"] * max(1.0, (k - 1) / math.log(k))
        span = math.log(hi / lo)
        cells, res = pairs * (hi * hi - lo * lo) / (2 * span), pairs * 2 * (hi - lo) / span
    else:
        pairs = case["pairs"]
        cells, res = pairs * _mean_square(case["median"]), 2.0 * pairs * case["median"] * math.exp(SIGMA ** 2 / 2)
    rows = 0.0
    if case.get("output", "alignment" if kind == "long" else "score") == "alignment":
        rows = 2.0 * pairs * math.sqrt(cells / pairs) * 1.1
    return {"bytes": res + 24.0 * pairs + 32.0 * pairs + rows, "flops": OPS_PER_CELL * cells}


# ---- the same results in plain numpy or torch ---------------------------------

_BLOSUM = None


def _blosum62():
    """BLOSUM62 over 'A'..'Z' (the published table; J, O and U score as X)."""
    global _BLOSUM
    if _BLOSUM is None:
        order = "ARNDCQEGHILKMFPSTWYVBZX"
        half = """4 -1 5 -2 0 6 -2 -2 1 6 0 -3 -3 -3 9 -1 1 0 0 -3 5 -1 0 0 2 -4 2 5 0 -2 0 -1 -3 -2 -2 6
        -2 0 1 -1 -3 0 0 -2 8 -1 -3 -3 -3 -1 -3 -3 -4 -3 4 -1 -2 -3 -4 -1 -2 -3 -4 -3 2 4
        -1 2 0 -1 -3 1 1 -2 -1 -3 -2 5 -1 -1 -2 -3 -1 0 -2 -3 -2 1 2 -1 5
        -2 -3 -3 -3 -2 -3 -3 -3 -1 0 0 -3 0 6 -1 -2 -2 -1 -3 -1 -1 -2 -2 -3 -3 -1 -2 -4 7
        1 -1 1 0 -1 0 0 0 -1 -2 -2 0 -1 -2 -1 4 0 -1 0 -1 -1 -1 -1 -2 -2 -1 -1 -1 -1 -2 -1 1 5
        -3 -3 -4 -4 -2 -2 -3 -2 -2 -3 -2 -3 -1 1 -4 -3 -2 11 -2 -2 -2 -3 -2 -1 -2 -3 2 -1 -1 -2 -1 3 -3 -2 -2 2 7
        0 -3 -3 -3 -1 -2 -2 -3 -3 3 1 -2 1 -1 -2 -2 0 -3 -1 4
        -2 -1 3 4 -3 0 1 -1 0 -3 -4 0 -3 -3 -2 0 -1 -4 -3 -3 4
        -1 0 0 1 -3 3 4 -2 0 -3 -3 1 -1 -3 -1 0 -1 -3 -2 -2 1 4
        0 -1 -1 -1 -2 -1 -1 -1 -1 -1 -1 -1 -1 -1 -2 0 0 -2 -1 -1 -1 -1 -1"""
        vals = [int(v) for v in half.split()]
        t = np.zeros((26, 26), dtype=np.int64)
        at = [ord(c) - 65 for c in order]
        k = 0
        for r in range(len(order)):
            for c in range(r + 1):
                t[at[r], at[c]] = t[at[c], at[r]] = vals[k]
                k += 1
        x = ord("X") - 65
        for letter in "JOU":
            u = ord(letter) - 65
            t[u, :] = t[x, :]
            t[:, u] = t[:, x]
        for p in "JOUX":
            for q in "JOUX":
                t[ord(p) - 65, ord(q) - 65] = t[x, x]
        _BLOSUM = t
    return _BLOSUM


def _exact_pair(a, b, matrix, gap_open, gap_extend, mode, output):
    """One pair by anti-diagonals in int64, then the walk from its end cell."""
    x = np.frombuffer(a, dtype=np.uint8).astype(np.int64) - 65
    y = np.frombuffer(b, dtype=np.uint8).astype(np.int64) - 65
    if matrix == "blosum62":
        table = _blosum62()
    else:
        table = np.where(np.eye(26, dtype=bool), 2, -3).astype(np.int64)
    m, n = len(x), len(y)
    go, ge, local = gap_open, gap_extend, mode == "local"
    oe, low = go + ge, -(1 << 40)
    edge = (lambda k: 0) if local else (lambda k: 0 if k == 0 else -(go + k * ge))
    # Row index i on a diagonal d = i + j; the arrays hold i = 0..m.
    H1 = np.full(m + 1, low, dtype=np.int64)  # diagonal d - 1
    H2 = H1.copy()                            # diagonal d - 2
    E, F = H1.copy(), H1.copy()               # of diagonal d - 1
    H1[0] = 0
    bits = np.zeros((m + 1, n + 1), dtype=np.uint8)
    best = (0, 0, 0)
    for d in range(1, m + n + 1):
        lo, hi = max(1, d - n), min(m, d - 1)
        H, E0, F0 = np.full(m + 1, low, dtype=np.int64), np.full(m + 1, low, dtype=np.int64), np.full(m + 1, low, dtype=np.int64)
        if d <= n:
            H[0] = edge(d)
        if d <= m:
            H[d] = edge(d)
        if lo <= hi:
            i = np.arange(lo, hi + 1)
            j = d - i
            eo, fo = H1[i] - oe, H1[i - 1] - oe
            e, f = np.maximum(E[i] - ge, eo), np.maximum(F[i - 1] - ge, fo)
            dd = H2[i - 1] + table[x[i - 1], y[j - 1]]
            h = np.maximum(np.maximum(dd, e), f)
            if local:
                h = np.maximum(h, 0)
            way = np.where(h == dd, 0, np.where(h == e, 1, 2))
            if local:
                way = np.where(h == 0, 3, way)
                k = int(h.max())
                at = int(np.flatnonzero(h == k)[0])
                if k > best[0] or (k == best[0] and k > 0 and (int(i[at]), int(j[at])) < best[1:]):
                    best = (k, int(i[at]), int(j[at]))
            bits[i, j] = way | ((e == eo) << 2) | ((f == fo) << 3)
            H[i], E0[i], F0[i] = h, e, f
            if d == m + n:
                last = int(h[-1])
        H2, H1, E, F = H1, H, E0, F0
    if local:
        score, i, j = best
    else:
        score, i, j = (last if m and n else edge(m + n)), m, n
    end = (i, j)
    ra, rb, state = [], [], 0
    while i > 0 or j > 0:
        if i == 0 or j == 0:
            if local:
                break
            if i == 0:
                ra.append(45), rb.append(y[j - 1] + 65)
                j -= 1
            else:
                ra.append(x[i - 1] + 65), rb.append(45)
                i -= 1
            continue
        v = int(bits[i, j])
        if state == 0:
            way = v & 3
            if way == 3:
                break
            if way == 0:
                ra.append(x[i - 1] + 65), rb.append(y[j - 1] + 65)
                i, j = i - 1, j - 1
            else:
                state = way
        elif state == 1:
            ra.append(45), rb.append(y[j - 1] + 65)
            state, j = (0 if v & 4 else 1), j - 1
        else:
            ra.append(x[i - 1] + 65), rb.append(45)
            state, i = (0 if v & 8 else 2), i - 1
    ra, rb = np.array(ra[::-1], dtype=np.uint8), np.array(rb[::-1], dtype=np.uint8)
    begin = (i, j) if output == "alignment" or not local or score <= 0 else (-1, -1)
    ident = int((ra == rb).sum()) if output != "score" else -1
    ncols = len(ra) if output != "score" else -1
    out = dict(score=score, a_begin=begin[0], a_end=end[0], b_begin=begin[1], b_end=end[1], n_ident=ident, n_cols=ncols,
               status=0)
    if output == "alignment":
        out["rows"] = np.concatenate([ra, rb])
    return out


def _exact_consensus(rows):
    """Per column: counts of the letters, the sums of each letter's row against
    all others, the first row with the highest sum."""
    nseq, ncols = rows.shape
    lut = np.full(256, 26, dtype=np.int64)
    lut[65:91] = np.arange(26)
    lut_d = torch.from_numpy(lut).to(rows.device)
    s = np.full((27, 27), -4, dtype=np.int64)
    s[:26, :26] = _blosum62()
    s[26, 26] = 1
    match = s > 0
    match[26, 26] = True
    same = np.arange(27)
    counts = torch.stack([(rows == c).sum(0) for c in range(65, 91)])
    counts = torch.cat([counts, (nseq - counts.sum(0))[None]]).cpu().numpy()
    sums = s @ counts - s[same, same][:, None]
    hits = match.astype(np.int64) @ counts - match[same, same].astype(np.int64)[:, None]
    top = np.where(counts > 0, sums, -(1 << 60)).max(0)
    win = torch.from_numpy((sums == top) & (counts > 0)).to(rows.device)
    line = np.zeros(ncols, dtype=np.uint8)
    matches = np.zeros(ncols, dtype=np.int32)
    todo = np.arange(ncols)
    step = 4096
    for r in range(0, nseq, step):  # the first row whose letter wins
        cls = lut_d[rows[r:r + step][:, torch.from_numpy(todo).to(rows.device)].long()]
        hit = win[:, torch.from_numpy(todo).to(rows.device)].gather(0, cls)
        first = hit.to(torch.uint8).argmax(0).cpu().numpy()
        found = hit.any(0).cpu().numpy()
        cls = cls.cpu().numpy()
        for q in np.flatnonzero(found):
            c = todo[q]
            matches[c] = hits[cls[first[q], q], c]
            line[c] = int(rows[r + int(first[q]), int(c)]) if matches[c] >= nseq / 2 else ord("?")
        todo = todo[~found]
        if not len(todo):
            break
    return [line, top.astype(np.int32), matches]


def exact(case, seed):
    if case["kind"] == "pair" and case["length"] <= 4000:
        a, b = _one_pair(case, seed)
        out = _exact_pair(a, b, **_params(case, _matrix(case["alphabet"])))
        if "rows" in out:
            out["rows"] = np.pad(out["rows"], (0, _rows_room(case) - len(out["rows"])))
        return out
    if case["kind"] == "consensus":
        return _exact_consensus(_alignment_rows(case, seed))
    return None  # hundreds of millions of cells, or thousands of scans of a matrix
