"""The tensor-core vote kernel (large dense predicts) against the oracle, bit for
bit: sample counts around its 256-sample tiles, clause rows around its
240-row tiles, classes of 8 clauses (a flush every 8 columns) and classes that
end inside a tile, rows whose bytes are not a multiple of a 256-literal step or
of 4 bytes, literal counts close to the row length (sums of odd integers far
above 2^13), clauses without literals, a tolerance beyond its exact range (the
other paths serve it), more samples than one launch takes; host and device
inputs, and again after the actions changed."""
import numpy as np
import pytest

import oracle as O
from test_gpu_parity import ref_table

pytestmark = pytest.mark.gpu


def _bits(rng, n, features, dens):
    b = rng.random((n, features)) < dens
    return np.packbits(np.concatenate([b, ~b], axis=1), axis=1, bitorder="little").ravel()


@pytest.mark.parametrize("kind,classes,features,clauses,dens,tol,sizes,fp4", [
    ("classifier", 3, 16384, 80, 0.9, 60000, (255, 256, 257), True),
    ("classifier", 30, 16384, 8, 0.0005, 20, (513,), True),
    ("classifier", 60, 1001, 248, 0.02, 40, (700, 1025), True),
    ("encoder", 29, 4099, 120, 0.004, 33, (500,), True),
    ("encoder", 3, 777, 2048, 0.02, 30, (1300,), True),
    ("classifier", 2, 524283, 8, 0.5, 60000, (1030,), True),
    ("classifier", 5, 2048, 240, 0.01, 70000, (400,), False),
])
def test_votes(tm, kind, classes, features, clauses, dens, tol, sizes, fp4):
    import torch
    rng = np.random.default_rng(classes * features)
    cfg = dict(type=kind, classes=classes, features=features, clauses=clauses, clause_tolerance=tol,
               clause_maximum=64, specificity=9.0)
    m = O.Machine(**cfg)
    k, tbl = ref_table(cfg)
    t = tm.create(k, tbl)
    t.stats_enable(True)
    row = m.info["action_chunks"] // (classes * clauses)
    for again in range(2):
        acts = np.packbits(rng.random(m.info["action_chunks"] * 8) < dens, bitorder="little")
        acts.reshape(-1, row)[::7] = 0  # clauses without literals
        m.load_state(actions=acts)
        t.import_state(actions=acts)
        for n in sizes:
            x = _bits(rng, n, features, 0.3)
            out, sc = m.predict(x, n, scores=True)
            assert np.array_equal(t.predict_scores(x, n), sc), n
            assert (t.stats()["predict_gemm"] == 2) == fp4
            got = t.predict(torch.tensor(x, device="cuda"), n)
            assert np.array_equal(got.cpu().numpy(), out.ravel()), n
        if features > 100000:
            break
    t.destroy()
