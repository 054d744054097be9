"""Epoch orders: a machine trained on n samples ends in the oracle's state only if
every epoch's order is the oracle's (samples by 64-bit Philox key, ties by index).
Sizes from one sample over the largest order sorted by one CTA (16,384) to
orders in global scratch, several epochs in one launch, several seeds in one
search round's graph."""
import numpy as np
import pytest

import oracle as O
from test_gpu_parity import ref_table, train_table

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,epochs", [(1, 3), (2, 2), (33, 70), (1023, 2), (16384, 2), (16385, 2),
                                      (70001, 3)])
def test_orders(tm, n, epochs):
    rng = np.random.default_rng(n)
    cfg = dict(type="classifier", classes=2, features=20, clauses=8, clause_tolerance=6,
               clause_maximum=9, specificity=4.0, target=7)
    b = rng.random((n, 20)) < 0.4
    x = np.packbits(np.concatenate([b, ~b], axis=1), axis=1, bitorder="little").ravel()
    y = (b[:, 0] ^ b[:, 3]).astype(np.int64)
    m = O.Machine(**cfg)
    m.train(x, n, epochs, labels=y, seed=n + 5)
    kind, tbl = ref_table(cfg, seed=n + 5)
    t = tm.create(kind, tbl)
    t.train(train_table(kind, dict(n=n, x=x, labels=y), epochs))
    a, s = t.export_state()
    assert np.array_equal(a, m.actions()) and np.array_equal(s, m.state())
    t.destroy()


def test_orders_of_a_search_round(tm):
    """Machines of different seeds and sizes, orders on both sides of the one-CTA
    limit in one graph: the automata equal those of machines trained alone."""
    rng = np.random.default_rng(4)
    ns = (500, 16500, 16384, 20000)
    b = rng.random((20000, 30)) < 0.4
    x = np.packbits(np.concatenate([b, ~b], axis=1), axis=1, bitorder="little")
    y = (b[:, 0] ^ b[:, 3]).astype(np.int64)
    tbl = dict(classes=2, features=30, clauses=16, clause_tolerance=6, clause_maximum=9,
               specificity=4.0, target=7, reusable=True)
    tt = [dict(samples=n, problems=x[:n].ravel(), solutions=y[:n], iterations=2) for n in ns]
    ms = [tm.create("classifier", dict(tbl, seed=i)) for i in range(4)]
    tm.train_batch_search(ms, tt, dict(samples=300, problems=x[:300].ravel(), solutions=y[:300]))
    for i, m in enumerate(ms):
        alone = tm.create("classifier", dict(tbl, seed=i))
        alone.train(tt[i])
        for p, q in zip(m.export_state(), alone.export_state()):
            assert np.array_equal(p, q), i
