"""Memory that a call can do without: when an allocation of it fails (the failure
is injected, tm_debug_fail_alloc), the call does the same work another way and
returns the same bytes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fails_at(tm, k):
    tm.lib().tm_debug_fail_alloc(k)


@pytest.mark.parametrize("ind", [False, True], ids=["dense", "individualized"])
def test_state_copies_without_staging(tm, ind):
    """Rows whose bytes are not whole 16-byte blocks are packed and unpacked in
    device memory of the call's own; without it they are copied row by row."""
    import torch
    rng = np.random.default_rng(5)
    n, hidden = 60, 5
    sizes = [41, 300, 77, 129, 8] if ind else [301] * hidden
    b = rng.random((n, max(sizes))) < 0.3
    blocks = [np.packbits(np.concatenate([b[:, :k], ~b[:, :k]], axis=1), axis=1,
                          bitorder="little").ravel() for k in (sizes if ind else sizes[:1])]
    tbl = dict(hidden=hidden, clauses=16, clause_tolerance=8, clause_maximum=30, specificity=5.0,
               target=10, reusable=True, seed=2)
    inp = dict(samples=n, sentences=np.concatenate(blocks), iterations=2,
               codes=rng.integers(0, 256, size=n).astype(np.uint8))
    if ind:
        tbl.update(individualized=True, feat_offsets=np.concatenate([[0], np.cumsum(sizes)]))
        inp["dim_offsets"] = np.cumsum([0] + [x.size for x in blocks]).astype(np.int64)
    else:
        tbl.update(visible=sizes[0])
    t = tm.create("encoder", tbl)
    t.train(inp)
    want = t.export_state()
    if not ind:
        part = torch.empty(sum(t.class_bytes(1, 4)), dtype=torch.uint8, device="cuda")
        t.export_classes(1, 4, part)
    for k in range(2):  # the actions' staging, the count planes'
        u = tm.create("encoder", tbl)
        try:
            _fails_at(tm, k)
            got = t.export_state()
            _fails_at(tm, k)
            u.import_state(actions=want[0], state=want[1])
            if not ind:
                mine = torch.zeros_like(part)
                _fails_at(tm, k)
                t.export_classes(1, 4, mine)
                _fails_at(tm, k)
                u.import_classes(1, 4, part)
        finally:
            _fails_at(tm, -1)
        assert all(np.array_equal(a, c) for a, c in zip(got, want))
        assert ind or torch.equal(mine, part)
        assert all(np.array_equal(a, c) for a, c in zip(u.export_state(), want))
        u.destroy()
