"""A tuned table's entries and the kernels they speak of: identity batches that
run on traceback planes follow the alignment entries, those that carry the counts
the identity entries."""
import json

import numpy as np
import pytest

from tweakseq_gb300 import aligner as A
from tweakseq_gb300 import build as B
from tweakseq_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built(tmp_path_factory):
    B.build()
    yield
    p = tmp_path_factory.mktemp("tune") / "empty.json"
    p.write_text(json.dumps({"entries": []}))
    A.load_tuning(str(p))


def test_identity_follows_the_entries_of_the_kernel_it_runs(tmp_path, monkeypatch):
    # Alignment entries: int32 lanes for short pairs, int16x2 for the rest (two
    # fill launches); identity entries: int16x2 for all (one).
    entries = [{"out": "identity", "lo": 0, "hi": 1 << 21, "G": 8, "R": 8, "i16": 1, "cta": 0, "gcups": 1.0},
               {"out": "alignment", "lo": 0, "hi": 200, "G": 8, "R": 8, "i16": 0, "cta": 0, "gcups": 1.0},
               {"out": "alignment", "lo": 200, "hi": 1 << 21, "G": 8, "R": 8, "i16": 1, "cta": 0, "gcups": 1.0}]
    p = tmp_path / "t.json"
    p.write_text(json.dumps({"entries": entries}))
    A.load_tuning(str(p))
    rng = np.random.default_rng(6)
    seqs = [W.random_protein(rng, 100 if k % 4 < 2 else 300).tobytes() for k in range(800)]
    ps = W._pairset_from_lists(seqs, [(2 * k, 2 * k + 1) for k in range(400)])

    def launches(output):
        with A.Batch(ps, output=output, autotune=True, use_graph=False) as b:
            b.run()
            return b.stats()["launches"]

    assert launches("identity") == launches("alignment")
    monkeypatch.setenv("TSQ_WAVE_BUDGET_BYTES", "1")
    assert launches("identity") == launches("alignment") - 2  # one fill fewer, and no walk
