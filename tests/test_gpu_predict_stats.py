"""What tm_stats says of a predict."""
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
