"""A search round's two train launches (rows of at most 32 words, and wider ones)
when both run one kernel: the narrow rows' picks (specificity 3: 333 of 1,000
literals) need more shared memory than the wide rows' (specificity 20: 100 of
2,000), so the kernel's limit has to hold for the larger of both.  The round's
automata equal those of machines trained alone, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [(4, 5), (4, 4), (3, 1), (0, 1)],
                         ids=["spec64", "wpt256", "warp", "cta"])
@pytest.mark.parametrize("narrow_first", [True, False], ids=["narrow_first", "wide_first"])
def test_one_kernel_for_narrow_and_wide_rows(tm, variant, narrow_first):
    rng = np.random.default_rng(8)
    n, nt, classes = 300, 40, 3
    b = rng.random((n + nt, 1000)) < 0.2
    y = (b[:, 0].astype(np.int64) + b[:, 5] + b[:, 9]) % classes

    def rows(f):
        return np.packbits(np.concatenate([b[:, :f], ~b[:, :f]], axis=1), axis=1,
                           bitorder="little")

    shapes = [(500, 3.0), (1000, 20.0)]
    if not narrow_first:
        shapes.reverse()
    tables, trains, tests = [], [], []
    for i, (f, s) in enumerate(shapes):
        x = rows(f)
        tables.append(dict(classes=classes, features=f, clauses=16, clause_tolerance=12,
                           clause_maximum=40, specificity=s, target=10, seed=i, reusable=True))
        trains.append(dict(samples=n, problems=x[:n].ravel(), solutions=y[:n], iterations=2))
        tests.append(np.ascontiguousarray(x[n:]).ravel())
    ms = [tm.create("classifier", t) for t in tables]
    ms[0].force_variant(*variant)
    ms[0].stats_enable(True)
    tm.train_batch_search(ms, trains, dict(samples=nt, problems_each=tests, solutions=y[n:]))
    assert (ms[0].stats()["train_mode"], ms[0].stats()["train_cpw"]) == variant
    for m, t, tr in zip(ms, tables, trains):
        alone = tm.create("classifier", t)
        alone.train(tr)
        for p, q in zip(m.export_state(), alone.export_state()):
            assert np.array_equal(p, q)
