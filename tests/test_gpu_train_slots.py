"""The train kernels of tm_train_wpt.cu at the edges of their row slots: each
configuration, pinned, against the oracle's state, bit for bit (whole numbers:
the tolerance is zero).  Row widths one word, a slot's last word, one past it,
rows whose last byte or word is partly used (with and without the reference's
unmasked 128-bit tail), several include bits, clauses that may gain literals
(clause_maximum above their literal counts), specificities below 1 (bits
picked four and more times), a target of 1 and negative samples always kept."""
import numpy as np
import pytest

import oracle as O
from test_gpu_parity import ref_table, train_table

pytestmark = pytest.mark.gpu

# features, configurations that hold 2 * features literals
ROWS = [
    (3, (5, 6, 7, 8, 4)),
    (508, (8, 5)),          # 32 words, a partly used last byte, 127 bytes
    (512, (8, 6)),          # 32 full words
    (513, (5, 7)),          # one word past the narrow slot
    (893, (7, 5)),          # 56 words, 224 bytes: the 128-bit tail
    (897, (6, 5)),          # one word past the 56-word slot
    (1021, (6, 5)),         # 64 words, 256 bytes, tail bits
    (1030, (4, 2)),
    (2041, (4, 2, 3)),      # 128 words
    (4093, (4, 2, 3)),      # 256 words
    (4099, (3, 1)),
    (8190, (3, 1)),         # 512 words
    (8200, (1,)),
    (16381, (1,)),          # 1,024 words
]


def _check(tm, cfg, inp, seed, pins, epochs=2):
    m = O.Machine(**cfg)
    m.train(inp["x"], inp["n"], epochs, labels=inp.get("labels"), codes=inp.get("codes"), seed=seed)
    kind, tbl = ref_table(cfg, seed=seed)
    for cpw in pins:
        t = tm.create(kind, tbl)
        if cpw:
            t.force_variant(4, cpw)
        t.stats_enable(True)
        t.train(train_table(kind, inp, epochs))
        if cpw:
            assert (t.stats()["train_mode"], t.stats()["train_cpw"]) == (4, cpw)
        a, s = t.export_state()
        assert np.array_equal(a, m.actions()), cpw
        assert np.array_equal(s, m.state()), cpw
        t.destroy()


def _rows(n, features, rng, density=0.1):
    b = rng.random((n, features)) < density
    return np.packbits(np.concatenate([b, ~b], axis=1), axis=1, bitorder="little").ravel()


@pytest.mark.parametrize("features,pins", ROWS, ids=[str(r[0]) for r in ROWS])
def test_row_widths(tm, features, pins):
    rng = np.random.default_rng(features)
    n = 150
    cfg = dict(type="classifier", classes=3, features=features, clauses=24, clause_tolerance=16,
               clause_maximum=40, specificity=9.0, target=14)
    _check(tm, cfg, dict(n=n, x=_rows(n, features, rng),
                         labels=rng.integers(0, 3, size=n).astype(np.int64)), 17, pins)


@pytest.mark.parametrize("include_bits,maximum,specificity,target", [
    (2, 30, 6.0, 12),
    (3, 100000, 6.0, 12),    # clauses gain literals
    (1, 100000, 3.0, 1),
    (1, 30, 0.5, 30),        # bits picked four and more times
    (8, 30, 0.7, 8),         # every plane counts for inclusion
])
@pytest.mark.parametrize("features,pins", [(301, (5, 6, 7, 8)), (1100, (2, 3, 4)), (4500, (1, 3))],
                         ids=["301", "1100", "4500"])
def test_feedback_options(tm, features, pins, include_bits, maximum, specificity, target):
    rng = np.random.default_rng(features + include_bits)
    n = 90
    codes = rng.integers(0, 256, size=n).astype(np.uint8)
    cfg = dict(type="encoder", classes=5, features=features, clauses=16, clause_tolerance=12,
               clause_maximum=maximum, include_bits=include_bits, specificity=specificity,
               target=target)
    _check(tm, cfg, dict(n=n, x=_rows(n, features, rng, 0.4), codes=codes), 23, pins)


@pytest.mark.parametrize("features,classes,clauses", [
    (1500, 10, 760),   # 950 units of 94-word rows: 128-word slots
    (2048, 10, 760),   # 128 words, the slot's last
    (768, 10, 760),    # 48 words, the slot's last
    (384, 10, 760),    # 24 words, the slot's last
    (397, 10, 760),    # 25 words, one past it
    (1500, 2, 40),     # 10 units: timed against the speculative kernel
    (16384, 3, 16),    # 1,024 words
])
def test_choices_without_pin(tm, features, classes, clauses):
    rng = np.random.default_rng(classes)
    n = 60
    cfg = dict(type="classifier", classes=classes, features=features, clauses=clauses,
               clause_tolerance=16, clause_maximum=50, specificity=11.0, target=20, negative=1.0)
    _check(tm, cfg, dict(n=n, x=_rows(n, features, rng),
                         labels=rng.integers(0, classes, size=n).astype(np.int64)), 3, (0,))
