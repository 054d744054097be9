"""Low specificities: bits that one Type Ib clause picks four times and more (the
overflow entries of tm_train_wpt.cu), in each row slot and in both forms of the
kernels, bit for bit against the oracle: a mean of 0.4 to 3 picks per bit, so
that clauses hold none, a few and hundreds of entries, bits are listed twice and
three times, and entries lie in every warp's words.  And the time of such a
launch beside another kernel's."""
import numpy as np
import pytest

import oracle as O
from test_gpu_parity import ref_table, train_table

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("specificity", [0.33, 1.2, 2.6])
@pytest.mark.parametrize("features,pins", [
    (24, (8, 5)), (380, (8, 7)), (512, (8, 6)), (890, (7, 5)), (1024, (6, 5)),
    (2048, (4, 2)), (4093, (4, 2, 3)), (8190, (3, 1)), (16384, (1,)), (1500, (0,)), (700, (0,))])
def test_overflow_entries(tm, features, pins, specificity):
    rng = np.random.default_rng(features)
    n, classes = 60, 3
    # (98,304 picks' entries fit no block's shared memory beside the largest slot)
    specificity = max(specificity, features / 20480)
    b = rng.random((n, features)) < 0.3
    x = np.packbits(np.concatenate([b, ~b], axis=1), axis=1, bitorder="little").ravel()
    y = rng.integers(0, classes, size=n).astype(np.int64)
    cfg = dict(type="classifier", classes=classes, features=features, clauses=16,
               clause_tolerance=12, clause_maximum=60, specificity=specificity, target=12,
               negative=1.0)
    m = O.Machine(**cfg)
    m.train(x, n, 2, labels=y, seed=9)
    kind, tbl = ref_table(cfg, seed=9)
    for pin in pins:
        t = tm.create(kind, tbl)
        if pin:
            t.force_variant(4, pin)
        t.stats_enable(True)
        t.train(train_table(kind, dict(n=n, x=x, labels=y), 2))
        assert t.stats()["train_mode"] == 4
        a, s = t.export_state()
        assert np.array_equal(a, m.actions()) and np.array_equal(s, m.state()), pin
        t.destroy()


def test_low_specificity_is_not_slower_than_the_cta_kernel(tm):
    """800 units of 24,000 literals at specificity 1.2 (250 entries per clause):
    the chosen kernel against the one-CTA kernel with the count planes in global
    memory, its closest relative (0.3 of its time; 2.2 when every entry was
    subtracted from every word)."""
    rng = np.random.default_rng(1)
    n, classes, features = 400, 10, 12000
    b = rng.random((n, features)) < 0.2
    x = np.packbits(np.concatenate([b, ~b], axis=1), axis=1, bitorder="little").ravel()
    t = tm.create("classifier", dict(classes=classes, features=features, clauses=640,
                                     clause_tolerance=64, clause_maximum=64, specificity=1.2,
                                     target=300, reusable=True, seed=3))
    t.stats_enable(True)
    inp = dict(samples=n, problems=x, solutions=rng.integers(0, classes, size=n).astype(np.int64),
               iterations=1)

    def best():
        t.train(inp)
        ms = []
        for _ in range(3):
            before = t.stats()["train_kernel_ms"]
            t.train(inp)
            ms.append(t.stats()["train_kernel_ms"] - before)
        return min(ms)

    chosen = best()
    assert t.stats()["train_mode"] == 4
    t.force_variant(1, 1)
    assert chosen < best()
