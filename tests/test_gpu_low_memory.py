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


def _clauses_of(tm, classes, features, clauses, literals, seed):
    """A machine whose clauses include `literals` literals each, and byte rows."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    t = tm.create("classifier", dict(classes=classes, features=features, clauses=clauses,
                                     clause_tolerance=20, clause_maximum=64, specificity=9.0,
                                     reusable=False))
    t.stats_enable(True)
    ab, sb = t.class_bytes(0, classes)
    acts = torch.zeros(classes * clauses, ab // (classes * clauses) * 8, dtype=torch.bool,
                       device="cuda")
    at = torch.randint(0, 2 * features, (classes * clauses, literals), generator=g, device="cuda")
    acts.scatter_(1, at, True)
    w = 1 << torch.arange(8, device="cuda", dtype=torch.int32)
    buf = torch.zeros(ab + sb, dtype=torch.uint8, device="cuda")
    buf[:ab] = (acts.view(classes * clauses, -1, 8).int() * w).sum(2).to(torch.uint8).reshape(-1)
    x = torch.randint(0, 256, (400, features // 4), generator=g, device="cuda", dtype=torch.uint8)
    x |= torch.randint(0, 256, x.shape, generator=g, device="cuda", dtype=torch.uint8)
    torch.cuda.synchronize()

    def fresh():  # a new state of the same automata: nothing derived is left
        t.import_classes(0, classes, buf)
    return t, x.cpu().numpy(), fresh


@pytest.mark.parametrize("n,literals", [(8, 20), (400, 20), (400, 700)],
                         ids=["few", "lists", "tensor"])
def test_predict_without_its_copies_of_the_actions(tm, n, literals):
    """Literal lists, the samples' slices, the 4-bit copies of actions and samples:
    a predict that cannot have them returns the same sums another way, and the
    next state uses them again."""
    t, x, fresh = _clauses_of(tm, 8, 8192, 4096, literals, n + literals)
    x = x[:n].ravel()
    fresh()
    want = t.predict_scores(x, n)
    want = t.predict_scores(x, n)  # (small requests: lists from the second on)
    t.destroy()
    refused = 0
    for k in range(12):
        t, _, fresh = _clauses_of(tm, 8, 8192, 4096, literals, n + literals)
        fresh()
        if n <= 32:
            assert np.array_equal(t.predict_scores(x, n), want)
        _fails_at(tm, k)
        try:
            got = t.predict_scores(x, n)
        except tm.TsetlinError as e:
            # host rows, vote sums and outputs: nothing else may be needed
            assert n > 32 and "memory" in str(e).lower()
            assert any(w in str(e) for w in ("sums", "raw", "outc", "m->x")), str(e)
            refused += 1
        else:
            assert np.array_equal(got, want), k
        finally:
            _fails_at(tm, -1)
        assert np.array_equal(t.predict_scores(x, n), want), k
        t.destroy()
    assert refused <= 4


def test_search_round_without_its_holdout_copies(tm):
    """The holdout of a large machine as 4-bit floats, and its actions: without them
    the round scores it with the bitwise kernel, to the same scores."""
    rng = np.random.default_rng(3)
    n, nt, classes, features = 200, 1200, 8, 2000
    b = rng.random((n + nt, features)) < 0.1
    y = (b[:, 0].astype(np.int64) + 2 * b[:, 7] + 4 * b[:, 11]) % classes
    x = np.packbits(np.concatenate([b, ~b], axis=1), axis=1, bitorder="little")
    tbl = dict(classes=classes, features=features, clauses=256, clause_tolerance=20,
               clause_maximum=40, specificity=9.0, target=30, reusable=True, seed=4)

    def run(k):
        t = tm.create("classifier", tbl)  # 2.5e8 tests of the holdout
        t.stats_enable(True)
        _fails_at(tm, k)
        try:
            r = tm.train_batch_search(
                [t], [dict(samples=n, problems=x[:n].ravel(), solutions=y[:n], iterations=2)],
                dict(samples=nt, problems=x[n:].ravel(), solutions=y[n:]))
        except tm.TsetlinError as e:
            assert "memory" in str(e).lower()
            return str(e)
        finally:
            _fails_at(tm, -1)
        launches = t.stats()["kernel_launches"]
        t.destroy()
        return [np.asarray(r["scores"]), np.asarray(r["best"])], launches

    run(-1)  # the tuner times its choices once
    want, usual = run(-1)
    fewer = 0
    for k in range(24):
        got = run(k)
        if isinstance(got, str):
            assert "search_x4" not in got and "search_act4" not in got, got
            continue
        assert all(np.array_equal(a, c) for a, c in zip(got[0], want)), k
        fewer += got[1] < usual
    assert fewer == 2  # the bitwise kernel is one launch an epoch, not two


def test_orders_one_after_another(tm):
    """Scratch for several large epoch orders at once (20,000 samples, three epochs):
    with room for one they run in turn."""
    rng = np.random.default_rng(6)
    n = 20000
    b = rng.random((n, 20)) < 0.4
    x = np.packbits(np.concatenate([b, ~b], axis=1), axis=1, bitorder="little").ravel()
    tbl = dict(classes=2, features=20, clauses=8, clause_tolerance=6, clause_maximum=9,
               specificity=4.0, target=7, reusable=True, seed=1)
    inp = dict(samples=n, problems=x, solutions=(b[:, 0] ^ b[:, 3]).astype(np.int64), iterations=3)
    t = tm.create("classifier", tbl)
    t.train(inp)
    want = t.export_state()
    t.destroy()
    for k in range(12):
        t = tm.create("classifier", tbl)
        _fails_at(tm, k)
        try:
            t.train(inp)
        except tm.TsetlinError as e:
            assert "memory" in str(e).lower() and "perm_scratch" not in str(e), str(e)
        else:
            assert all(np.array_equal(a, c) for a, c in zip(t.export_state(), want)), k
        finally:
            _fails_at(tm, -1)
        t.destroy()
