"""Which train kernel runs: a call that launches once per epoch (an `each`
callback, a batch with one, machines of a batch that end early) keeps the
word-per-thread kernels (train_mode 4) after its first epoch, whether the tuner
timed two of them or had one choice, and ends in the state of a call that runs
all epochs at once."""
import numpy as np
import pytest

import oracle as O
from test_gpu_parity import ref_table, train_table

pytestmark = pytest.mark.gpu

SHAPES = [
    (10, 784, 760),    # 950 units: one choice
    (10, 16384, 64),   # 1,024 words: one choice
    (10, 784, 64),     # 80 units: two choices, timed
]
IDS = ["units950", "words1024", "units80"]


def _table(classes, features, clauses, seed=1):
    return dict(classes=classes, features=features, clauses=clauses, clause_tolerance=16,
                clause_maximum=50, specificity=11.0, target=20, reusable=True, seed=seed)


def _inputs(classes, features, n=120):
    rng = np.random.default_rng(classes * features)
    b = rng.random((n, features)) < 0.1
    x = np.packbits(np.concatenate([b, ~b], axis=1), axis=1, bitorder="little").ravel()
    return dict(samples=n, problems=x, solutions=rng.integers(0, classes, size=n).astype(np.int64),
                iterations=3)


@pytest.mark.parametrize("autotune", [1, 2])
@pytest.mark.parametrize("shape", SHAPES, ids=IDS)
def test_each_epoch_keeps_the_kernel(tm, shape, autotune):
    inp = _inputs(shape[0], shape[1])
    t = tm.create("classifier", _table(*shape))
    t.set_autotune(autotune)
    t.stats_enable(True)
    seen = []

    def each(epoch):
        st = t.stats()
        seen.append((st["train_mode"], st["train_cpw"], st["train_autotuned"]))
        return True

    t.train(dict(inp, each=each))
    assert len(seen) == 3 and seen[0][0] == 4 and set(seen) == {seen[0]}, seen
    assert seen[0][2] == 1
    once = tm.create("classifier", _table(*shape))
    once.set_autotune(0)
    once.train(inp)
    for a, b in zip(t.export_state(), once.export_state()):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("shape", SHAPES, ids=IDS)
def test_batch_epochs_keep_the_kernel(tm, shape):
    inp = _inputs(shape[0], shape[1])
    ms = [tm.create("classifier", _table(*shape, seed=i)) for i in range(3)]
    ms[0].stats_enable(True)
    seen = []

    def each(epoch):
        seen.append(ms[0].stats()["train_mode"])

    # machine i trains i + 1 epochs: each launch has fewer units than the one before
    tm.train_batch(ms, [dict(inp, iterations=i + 1) for i in range(3)], each=each)
    assert seen == [4, 4, 4]
    for i, m in enumerate(ms):
        once = tm.create("classifier", _table(*shape, seed=i))
        once.set_autotune(0)
        once.train(dict(inp, iterations=i + 1))
        for a, b in zip(m.export_state(), once.export_state()):
            assert np.array_equal(a, b)


def test_few_units_get_more_threads_where_that_is_faster(tm):
    """800 units of 94-word rows, 5.4 per SM: two warps per unit (configuration 4)
    take 0.75 of the time of one (10) or of eight samples at once (9)."""
    rng = np.random.default_rng(2)
    n, hidden, visible = 2000, 10, 1500
    b = rng.random((n, visible)) < 0.2
    x = np.packbits(np.concatenate([b, ~b], axis=1), axis=1, bitorder="little").ravel()
    t = tm.create("encoder", dict(hidden=hidden, visible=visible, clauses=640, clause_tolerance=64,
                                  clause_maximum=64, specificity=4.0, target=30, reusable=True,
                                  seed=3))
    t.set_autotune(2)
    t.stats_enable(True)
    t.train(dict(samples=n, sentences=x, codes=rng.integers(0, 256, size=2 * n).astype(np.uint8),
                 iterations=1))
    st = t.stats()
    assert (st["train_mode"], st["train_cpw"], st["train_autotuned"]) == (4, 4, 1)


@pytest.mark.parametrize("features,config", [
    (880, 7), (912, 7), (1024, 7), (1024, 6), (1024, 5), (4096, 4), (8192, 3), (4096, 2),
    (16384, 1)])
def test_pinned_configurations_hold_the_widest_rows_they_held(tm, features, config):
    """Rows of 55 to 1,024 words under the configurations whose numbers callers may
    have pinned: 7 holds 64 words, also since its own slots have 56."""
    rng = np.random.default_rng(features)
    n, classes = 80, 3
    b = rng.random((n, features)) < 0.1
    x = np.packbits(np.concatenate([b, ~b], axis=1), axis=1, bitorder="little").ravel()
    y = rng.integers(0, classes, size=n).astype(np.int64)
    cfg = dict(type="classifier", classes=classes, features=features, clauses=16,
               clause_tolerance=12, clause_maximum=30, specificity=8.0, target=12)
    m = O.Machine(**cfg)
    m.train(x, n, 2, labels=y, seed=6)
    kind, tbl = ref_table(cfg, seed=6)
    t = tm.create(kind, tbl)
    t.force_variant(4, config)
    t.stats_enable(True)
    t.train(train_table(kind, dict(n=n, x=x, labels=y), 2))
    assert (t.stats()["train_mode"], t.stats()["train_cpw"]) == (4, config)
    a, s = t.export_state()
    assert np.array_equal(a, m.actions()) and np.array_equal(s, m.state())
    t.destroy()
