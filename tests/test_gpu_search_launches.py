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


_ROUND = """
import sys
sys.path[:0] = [%r, %r, %r]
import numpy as np
import santoku_tsetlin as tm
tol = int(sys.argv[1])
rng = np.random.default_rng(3)
n, nt, classes, features = 150, 1500, 8, 2000
b = rng.random((n + nt, features)) < 0.1
y = (b[:, 0].astype(np.int64) + 2 * b[:, 7] + 4 * b[:, 11]) %% classes
x = np.packbits(np.concatenate([b, ~b], axis=1), axis=1, bitorder="little")
ms = []
for i, clauses in enumerate((256, 400, 16)):  # 3.8e8, 6.0e8 and 2.4e7 tests of the holdout
    ms.append(tm.create("classifier", dict(
        classes=classes, features=features, clauses=clauses, clause_tolerance=tol,
        clause_maximum=40, specificity=9.0, target=30, reusable=True, seed=i)))
ms[0].stats_enable(True)
tr = dict(samples=n, problems=x[:n].ravel(), solutions=y[:n], iterations=3)
te = dict(samples=nt, problems=x[n:].ravel(), solutions=y[n:])
tm.train_batch_search(ms, [dict(tr, iterations=1)] * 3, te)  # tunes
ms[0].reset_stats()
r = tm.train_batch_search(ms, [tr] * 3, te, patience=3)
print("LAUNCHES", ms[0].stats()["kernel_launches"])
print("SCORES", np.asarray(r["scores"]).tolist(), np.asarray(r["final"]).tolist())
"""


def _round(switch, tol):
    import os
    import subprocess
    import sys
    here = os.path.dirname(os.path.abspath(__file__))
    root = os.path.dirname(here)
    code = _ROUND % (here, os.path.join(root, "lua-santoku-tsetlin_b200"),
                     os.path.join(root, "oracle"))
    r = subprocess.run([sys.executable, "-c", code, str(tol)],
                       env=dict(os.environ, TSETLIN_B200_GEMM=switch), capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    out = dict(ln.split(" ", 1) for ln in r.stdout.splitlines() if " " in ln)
    return int(out["LAUNCHES"]), out["SCORES"]


@pytest.mark.parametrize("tol", [20, 70000])
def test_holdout_of_large_machines_uses_the_tensor_cores(tol):
    """The holdout of the two large machines, by TSETLIN_B200_GEMM: off, the tiles of
    all three machines are one launch; int8 and fp8, and fp4 where the tolerance is
    beyond its range, two launches of the library's own per machine and epoch more
    (the products are cuBLASLt's).  The scores are the same."""
    off, scores = _round("off", tol)
    for switch in ("int8", "fp8", "fp4"):
        launches, got = _round(switch, tol)
        assert got == scores, switch
        assert launches >= off + 3 * 2 * 2, (switch, launches, off)
