"""Requests of 17 to 32 samples: small machines evaluate two groups of samples in
one launch (both halves of odd and even counts, classes and codes, rows of which
16, 15 and 8 fit a launch), larger machines and wider rows one after another;
calls in turn on one machine, since the launch leaves its sums and counters
cleared for the next.  Whole numbers against the oracle: the tolerance is zero."""
import numpy as np
import pytest

import oracle as O
from test_gpu_parity import ref_table

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,classes,features,clauses,launches", [
    ("classifier", 10, 784, 256, 1),
    ("encoder", 37, 693, 72, 1),
    ("classifier", 3, 16384, 8, 1),
    ("encoder", 9, 3, 8, 1),
    ("classifier", 2, 18432, 40, 1),     # 1,152 words: 16 rows in 72 KB
    ("classifier", 2, 18500, 40, None),  # 1,160 words: 12 rows a launch
    ("classifier", 2, 24000, 40, None),
    ("classifier", 10, 784, 472, 1),     # 4,720 clauses, the most
    ("classifier", 10, 784, 480, 2),
])
def test_two_groups(tm, kind, classes, features, clauses, launches):
    import torch
    rng = np.random.default_rng(features + clauses)
    cfg = dict(type=kind, classes=classes, features=features, clauses=clauses, clause_tolerance=30,
               clause_maximum=64, specificity=9.0)
    m = O.Machine(**cfg)
    k, tbl = ref_table(cfg)
    t = tm.create(k, tbl)
    t.stats_enable(True)
    acts = np.packbits(rng.random(m.info["action_chunks"] * 8) < 20.0 / features,
                       bitorder="little")
    m.load_state(actions=acts)
    t.import_state(actions=acts)
    b = rng.random((32, features)) < 0.3
    x = np.packbits(np.concatenate([b, ~b], axis=1), axis=1, bitorder="little")
    t.predict(x[:1].ravel(), 1)  # literal counts
    for n in (17, 32, 16, 25, 31, 24, 1, 18):
        rows = x[:n].ravel()
        out, sc = m.predict(rows, n, scores=True)
        before = t.stats()["kernel_launches"]
        assert np.array_equal(t.predict_scores(rows, n), sc), n
        if n > 16 and launches:
            assert t.stats()["kernel_launches"] - before == launches, n
        got = t.predict(torch.tensor(rows, device="cuda"), n)
        assert np.array_equal(got.cpu().numpy().ravel(), np.asarray(out).ravel()), n
    t.destroy()
