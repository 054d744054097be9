"""Predicts of at most 32 samples of dense machines (one launch from byte rows to
outputs) against the oracle, bit for bit: every sample count with a kernel of
its own and across the 16-sample launches, rows whose bytes start unaligned,
rows of one word and rows too wide for 16 of them to be staged at once, clause
counts that leave odd remainders to a warp, ties, codes whose last byte is
partly used; inputs from host memory and from the GPU; calls in a row (the vote
sums are left at zero)."""
import numpy as np
import pytest

import oracle as O
from test_gpu_parity import ref_table

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,classes,features,clauses,dens", [
    ("classifier", 3, 3, 8, 0.3),
    ("classifier", 10, 61, 24, 0.05),
    ("classifier", 37, 100, 8, 0.05),
    ("encoder", 13, 784, 40, 0.02),
    ("encoder", 70, 2001, 16, 0.01),
    ("classifier", 5, 60001, 8, 0.0005),
    ("classifier", 2, 512, 4096, 0.02),
])
def test_few(tm, kind, classes, features, clauses, dens):
    import torch
    rng = np.random.default_rng(features)
    cfg = dict(type=kind, classes=classes, features=features, clauses=clauses, clause_tolerance=20,
               clause_maximum=30, specificity=9.0)
    m = O.Machine(**cfg)
    acts = np.packbits(rng.random(m.info["action_chunks"] * 8) < dens, bitorder="little")
    m.load_state(actions=acts)
    k, tbl = ref_table(cfg)
    t = tm.create(k, tbl)
    t.import_state(actions=acts)
    for n in (1, 2, 3, 4, 5, 6, 7, 8, 9, 12, 13, 16, 17, 28, 32):
        b = rng.random((n, features)) < 0.3
        x = np.packbits(np.concatenate([b, ~b], axis=1), axis=1, bitorder="little").ravel()
        out, sc = m.predict(x, n, scores=True)
        assert np.array_equal(t.predict_scores(x, n), sc), n
        assert np.array_equal(t.predict(x, n), out.ravel()), n
        assert np.array_equal(t.predict(torch.tensor(x, device="cuda"), n).cpu().numpy(), out.ravel()), n
    t.destroy()
