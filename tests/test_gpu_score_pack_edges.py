"""The scoring and packing kernels at their edges, against the CPU restatements
(counts and bytes exact, doubles equal to the last bit: the tolerance is zero):
row widths around 32-bit words and unaligned rows, more counters than a CTA
keeps in shared memory, byte columns longer than a counter byte holds, fewer
threads than columns, device inputs, calls in a row on one scratch pool."""
import numpy as np
import pytest

import evaluator_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("features", [1, 3, 4, 7, 8, 15, 16, 17, 31, 32, 33, 63, 64, 65, 100, 1001])
@pytest.mark.parametrize("flip", [True, False])
@pytest.mark.parametrize("n", [1, 37])
def test_pack_widths(tm, features, flip, n):
    import torch
    rng = np.random.default_rng(features * 2 + flip)
    bits = rng.random((n, features)) < 0.4
    s, f = np.nonzero(bits)
    idx = (s * features + f).astype(np.int64)
    rng.shuffle(idx)
    idx = np.concatenate([idx, idx[:3], [-7, n * features, (1 << 33) + 5]]).astype(np.int64)
    want = R.bits_to_cvec(idx, n, features, flip)
    assert np.array_equal(tm.bits_to_cvec(idx, n, features, flip), want)
    got = tm.bits_to_cvec(torch.tensor(idx, device="cuda"), n, features, flip)
    assert np.array_equal(got.cpu().numpy(), want)


@pytest.mark.parametrize("features", [128, 256, 384, 1152, 127, 129])
@pytest.mark.parametrize("flip", [True, False])
def test_pack_aligned_rows(tm, features, flip):
    """Whole 16-byte rows, through fewer and more quads than a CTA; an output
    that is not 16-byte aligned."""
    import torch
    rng = np.random.default_rng(features)
    for n in (1, 3, 301):
        s, f = np.nonzero(rng.random((n, features)) < 0.1)
        idx = (s * features + f).astype(np.int64)
        want = R.bits_to_cvec(idx, n, features, flip)
        assert np.array_equal(tm.bits_to_cvec(idx, n, features, flip), want)
        dev = torch.tensor(idx, device="cuda")
        assert np.array_equal(tm.bits_to_cvec(dev, n, features, flip).cpu().numpy(), want)
        buf = torch.zeros(want.size + 16, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        out = buf[4:4 + want.size]
        tm._check(tm.lib().tm_bits_to_cvec(dev.data_ptr(), dev.numel(), n, features, int(flip), 1, 0,
                                           out.data_ptr()))
        assert np.array_equal(out.cpu().numpy(), want.ravel())
        assert not buf[:4].any() and not buf[4 + want.size:].any()


def test_pack_no_set_bits(tm):
    for flip in (True, False):
        want = R.bits_to_cvec(np.zeros(0, np.int64), 5, 45, flip)
        assert np.array_equal(tm.bits_to_cvec(np.zeros(0, np.int64), 5, 45, flip), want)


@pytest.mark.parametrize("n,hidden", [(2, 7), (3, 8), (5, 9), (70000, 3), (40, 12000), (3, 90001),
                                      (50, 255), (50, 256), (50, 257), (50, 1)])
def test_code_scores(tm, n, hidden):
    import torch
    rng = np.random.default_rng(n + hidden)
    nb = (hidden + 7) // 8
    e = rng.integers(0, 256, size=n * nb).astype(np.uint8)
    p = e ^ np.packbits(rng.random((n, nb * 8)) < 0.6, axis=1, bitorder="little").ravel()
    want = R.encoding_accuracy(p, e, n, hidden)
    assert tm.encoding_accuracy(p, e, n, hidden) == want
    assert tm.encoding_accuracy(torch.tensor(p, device="cuda"), torch.tensor(e, device="cuda"), n,
                                hidden) == want
    same = tm.encoding_accuracy(e, e, n, hidden)
    assert same == R.encoding_accuracy(e, e, n, hidden)


@pytest.mark.parametrize("n,classes", [(0, 3), (1, 2), (300, 5000), (50000, 2)])
def test_class_scores(tm, n, classes):
    rng = np.random.default_rng(classes)
    t = rng.integers(0, classes, size=n).astype(np.int64)
    p = np.where(rng.random(n) < 0.5, t, rng.integers(0, classes, size=n)).astype(np.int64)
    for _ in range(3):
        assert tm.class_accuracy(p, t, n, classes) == R.class_accuracy(p, t, n, classes)
