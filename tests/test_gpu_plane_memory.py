"""Device memory of identity calls: traceback planes are a workspace that gives
way -- to a call's own second try, to alignment calls of the same thread, and to
what others have left free."""
import threading

import numpy as np
import pytest

from tweakseq_gb300 import aligner as A
from tweakseq_gb300 import build as B

pytestmark = pytest.mark.gpu
GB = 1 << 30


@pytest.fixture(scope="module", autouse=True)
def built():
    B.build()


def on_own_thread(f):
    """Runs f on a thread of its own: the library's cached engines are the
    thread's, and go with it."""
    out = {}

    def run():
        try:
            out["value"] = f()
        except BaseException as e:  # noqa: BLE001 (handed to the caller)
            out["error"] = e

    t = threading.Thread(target=run)
    t.start()
    t.join()
    if "error" in out:
        raise out["error"]
    return out.get("value")


def free_bytes():
    import torch

    return torch.cuda.mem_get_info()[0]


def leave_free(keep):
    """A buffer that leaves `keep` bytes of device memory free."""
    import torch

    torch.cuda.empty_cache()
    return torch.empty(free_bytes() - keep, dtype=torch.uint8, device="cuda")


def equal_pairs(n, length):
    """n pairs of `length` residues out of one buffer, at shifting offsets."""
    rng = np.random.default_rng(length)
    seqs = np.frombuffer(b"ARNDCQEGHILKMFPSTWYV", dtype=np.uint8)[rng.integers(0, 20, length + 4096)]
    k = np.arange(n)
    return seqs, (k * 7) % 4096, np.full(n, length), (k * 7 + 3) % 4096, np.full(n, length)


def identity(pairs):
    return A.align_batch(pairs, output="identity").table


def test_second_try_releases_the_planes_of_the_first(monkeypatch):
    torch = pytest.importorskip("torch")
    pairs = equal_pairs(32768, 740)  # two chunks, 4.2 and 8.4 GB of planes

    def body():
        monkeypatch.setenv("TSQ_WAVE_BUDGET_BYTES", "1")
        want = identity(pairs)
        monkeypatch.delenv("TSQ_WAVE_BUDGET_BYTES")
        hold = leave_free(6 * GB)
        got = identity(pairs)
        left = free_bytes()
        del hold
        torch.cuda.empty_cache()
        assert np.array_equal(got, want)
        assert left > 4.5 * GB, left / GB

    on_own_thread(body)


def test_alignments_take_back_an_identity_calls_planes():
    torch = pytest.importorskip("torch")
    pairs = equal_pairs(32768, 500)  # 2.2 GB of planes in one chunk's engine, 4.4 in the other's
    rng = np.random.default_rng(5)
    a = np.frombuffer(b"ACGT", dtype=np.uint8)[rng.integers(0, 4, 92_000)]
    two = (a, [0, 0], [len(a)] * 2, [0, 0], [len(a)] * 2)  # 4.2 GB of planes each

    def body():
        identity(pairs)
        hold = leave_free(3 * GB)
        try:
            got = A.align_batch(two, matrix="dna", gap_open=5, gap_extend=2, output="alignment")
        finally:
            del hold
            torch.cuda.empty_cache()
        assert got.table["score"].tolist() == [2 * len(a)] * 2
        assert got.aln_a[0] == got.aln_b[1] == a.tobytes().decode()

    on_own_thread(body)


@pytest.mark.parametrize("form", ["one of a batch", "pair", "resident"])
def test_other_calls_take_back_an_identity_calls_planes(form):
    """4.2 GB of planes with 1.2 GB free and 6.6 GB in the identity call's engines."""
    torch = pytest.importorskip("torch")
    pairs = equal_pairs(32768, 500)
    rng = np.random.default_rng(6)
    a = np.frombuffer(b"ACGT", dtype=np.uint8)[rng.integers(0, 4, 92_000)]
    kw = dict(matrix="dna", gap_open=5, gap_extend=2, output="alignment")

    def align():
        if form == "pair":
            return A.align_pair(a.tobytes(), a.tobytes(), **kw)
        one = (a, [0], [len(a)], [0], [len(a)])
        if form == "one of a batch":
            return A.align_batch(one, **kw)[0]
        with A.Batch(one, use_graph=False, **kw) as b:
            b.run()
            return b.results()[0]

    def body():
        identity(pairs)
        hold = leave_free(int(1.2 * GB))
        try:
            got = align()
        finally:
            del hold
            torch.cuda.empty_cache()
        assert got.score == 2 * len(a) and got.aln_a == got.aln_b == a.tobytes().decode()

    on_own_thread(body)


@pytest.mark.parametrize("resident", [False, True])
def test_planes_take_a_share_of_what_is_free(resident, monkeypatch):
    torch = pytest.importorskip("torch")
    pairs = equal_pairs(32768, 500)  # 6.6 GB of planes

    def run():
        if not resident:
            return identity(pairs), free_bytes()
        with A.Batch(pairs, output="identity") as b:
            b.run()
            return b.results().table, free_bytes()

    def body():
        monkeypatch.setenv("TSQ_WAVE_BUDGET_BYTES", "1")
        want, _ = run()
        monkeypatch.delenv("TSQ_WAVE_BUDGET_BYTES")
        hold = leave_free(8 * GB)
        got, left = run()
        del hold
        torch.cuda.empty_cache()
        assert np.array_equal(got, want)
        assert left > 5 * GB, left / GB

    on_own_thread(body)
