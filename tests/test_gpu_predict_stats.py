"""What a machine says of its last predict: the path that evaluated it
(tm_predict_path), so that a test or a benchmark can tell them apart, and the
kernels' time (tm_stats)."""
import os
import subprocess
import sys

import numpy as np
import pytest

from test_gpu_low_memory import _clauses_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("literals", [20, 700], ids=["lists", "tensor"])
def test_kernel_time_has_no_host_copy_in_it(tm, literals):
    """20,000 samples of 4 KB from pageable memory take tens of milliseconds to copy,
    their evaluation about one."""
    import torch
    t, _, fresh = _clauses_of(tm, 4, 16384, 1024, literals, literals)
    fresh()
    n = 20000
    x = torch.randint(0, 256, (n * 4096,), dtype=torch.uint8, device="cuda")
    host = x.cpu().numpy()

    def took(rows):
        before = t.stats()["predict_kernel_ms"]
        got = t.predict(rows, n)
        return t.stats()["predict_kernel_ms"] - before, np.asarray(torch.as_tensor(got).cpu())

    took(x)
    from_device = [took(x) for _ in range(3)]
    from_host = [took(host) for _ in range(3)]
    assert np.array_equal(from_device[0][1], from_host[0][1])
    a, b = min(v[0] for v in from_device), min(v[0] for v in from_host)
    assert 0 < b < 1.5 * a, (a, b)
    t.destroy()


@pytest.mark.parametrize("classes,features,clauses,literals,n,path", [
    (4, 784, 64, 20, 1, "few"),
    (4, 784, 64, 20, 32, "few"),
    (4, 784, 64, 20, 33, "bitwise"),
    (10, 784, 256, 20, 400, "fp4"),          # 5e7 tests
    (4, 7152, 5008, 32, 129, "lists"),       # tiles of 4 words
    (3, 7156, 6504, 32, 129, "lists"),       # of 2
    (2, 14324, 4816, 32, 65, "lists"),       # of 1
    (2, 28660, 2480, 32, 100, "fp4"),        # rows too wide for lists
    (4, 4096, 8192, 300, 100, "fp4"),        # 1 literal in 27
    (4, 16384, 4096, 1500, 100, "fp4"),      # more literals than a counter holds
])
def test_path_by_shape(tm, classes, features, clauses, literals, n, path):
    t, x, fresh = _clauses_of(tm, classes, features, clauses, literals, features)
    assert t.predict_path() == "none"
    fresh()
    t.predict(x[:n].ravel(), n)
    assert t.predict_path() == path
    t.predict_scores(x[:n].ravel(), n)
    assert t.predict_path() == path
    t.reset_stats()
    assert t.predict_path() == "none"
    t.destroy()


def test_small_requests_move_to_lists_and_back(tm):
    """Machines beyond L2: the second request of three samples or more in a state
    reads lists, one or two samples never do, a new state starts over."""
    t, x, fresh = _clauses_of(tm, 8, 8192, 4096, 30, 5)
    for _ in range(2):
        fresh()
        seen = []
        for n in (2, 5, 1, 3, 32, 2):
            t.predict(x[:n].ravel(), n)
            seen.append(t.predict_path())
        assert seen == ["few", "few", "few", "lists", "lists", "few"]
    t.destroy()


def test_path_of_an_individualized_machine(tm):
    rng = np.random.default_rng(1)
    sizes = [700, 900]
    t = tm.create("encoder", dict(hidden=2, clauses=1600, clause_tolerance=8, clause_maximum=30,
                                  specificity=5.0, individualized=True, reusable=True,
                                  feat_offsets=np.concatenate([[0], np.cumsum(sizes)])))
    n = 400
    blocks = [rng.integers(0, 256, size=n * (k // 4), dtype=np.uint8) for k in sizes]
    off = np.cumsum([0] + [b.size for b in blocks]).astype(np.int64)
    t.predict(np.concatenate(blocks), off, n)
    assert t.predict_path() == "bitwise"
    t.destroy()


@pytest.mark.parametrize("switch,path", [("int8", "int8"), ("fp8", "fp8"), ("off", "bitwise"),
                                         ("fp4", "lists")])
def test_path_by_switch(switch, path):
    here = os.path.dirname(os.path.abspath(__file__))
    code = """
import sys
sys.path[:0] = [%r, %r, %r]
import santoku_tsetlin as tm
from test_gpu_low_memory import _clauses_of
t, x, fresh = _clauses_of(tm, 4, 7152, 5008, 32, 1)
fresh()
t.predict(x[:129].ravel(), 129)
print("PATH", t.predict_path())
""" % (here, os.path.join(os.path.dirname(here), "lua-santoku-tsetlin_b200"),
       os.path.join(os.path.dirname(here), "oracle"))
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, TSETLIN_B200_GEMM=switch),
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    assert "PATH " + path in r.stdout
