"""Large predicts over literal lists, bit for bit: each tile width (rows up to
447, 895 and 1,791 words and the next), rows whose bytes are no
multiple of 4, sample counts around a tile, clause counts that fill no group of
32, lists of 0, 15, 16, 17 and more literals, clauses above and below the
tolerance, counters of 7 and of 10 bits (127 and 128 literals), sums beyond the
4,095 kept between flushes, a machine with one clause too long for a counter and
one with rows too dense (the tensor cores serve them); again after the actions
changed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _unpack(b, rows):
    import torch
    sh = torch.arange(8, device="cuda", dtype=torch.uint8)
    return ((b.view(rows, -1).unsqueeze(2) >> sh) & 1).reshape(rows, -1)


def _want(acts, x, classes, clauses, n, bits, tol):
    """Vote sums by the definition (capi.c:97-161), counts exact in fp64."""
    import torch
    off = 1.0 - _unpack(x, n)[:, :bits].double()
    out = torch.zeros(n, classes, dtype=torch.int64, device="cuda")
    for h, a in enumerate(acts.view(classes, -1)):
        a = _unpack(a.contiguous(), clauses)[:, :bits].double()
        L = a.sum(1)
        cap = torch.where((L == 0) | (L > tol), torch.full_like(L, tol), L)
        v = (cap - off @ a.T).clamp(min=0).long()
        out[:, h] = v[:, 0::2].sum(1) - v[:, 1::2].sum(1)
    return out


CASES = [
    # classes, features, clauses, tolerance, literal counts, samples, lists
    (4, 7152, 5008, 64, (0, 15, 16, 17, 32), (33, 128, 129), True),   # 447 words, 4-word tiles
    (3, 7153, 6504, 20, (30, 64, 100, 127), (200,), True),            # 448 words, 2-word tiles
    (3, 14320, 3304, 1000, (5, 128, 300), (63, 65), True),            # 895 words, 2-word tiles
    (2, 14321, 4816, 40, (3, 127, 128, 400), (65,), True),            # 896 words, 1-word tiles
    (2, 28656, 2480, 16, (60, 20), (100,), True),                     # 1,791 words
    (2, 28657, 2480, 16, (60, 20), (100,), False),                    # 1,792 words: too wide
    (2, 20000, 3400, 64, (10,), (40,), "long"),                       # one clause of 1,024
    (4, 4096, 8192, 64, (300,), (40,), False),                        # 1 literal in 27
    (37, 2001, 3608, 30, (9, 33), (300,), True),                      # narrow rows, many classes
]


@pytest.mark.parametrize("classes,features,clauses,tol,counts,sizes,lists", CASES,
                         ids=["%dx%d" % (c[1], c[2]) for c in CASES])
def test_lists(tm, classes, features, clauses, tol, counts, sizes, lists):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(features)
    t = tm.create("classifier", dict(classes=classes, features=features, clauses=clauses,
                                     clause_tolerance=tol, clause_maximum=64, specificity=9.0,
                                     reusable=False))
    t.stats_enable(True)
    bits, row = 2 * features, (2 * features + 7) // 8
    w = (1 << torch.arange(8, device="cuda", dtype=torch.int32))
    for again in range(2):
        acts = []
        for h in range(classes):
            a = torch.zeros(clauses, row * 8, dtype=torch.bool, device="cuda")
            n = torch.tensor(counts, device="cuda").repeat(clauses + 1)[again:again + clauses]
            k = int(max(counts))
            at = torch.rand(clauses, bits, generator=g, device="cuda").topk(k, dim=1).indices
            a.scatter_(1, at, torch.arange(k, device="cuda") < n[:, None])
            if lists == "long" and h == 1:
                a[clauses // 2, 5:1029] = True
                a[clauses // 2, 1029:] = False
                a[clauses // 2, :5] = False
            acts.append((a.view(clauses, row, 8).int() * w).sum(2).to(torch.uint8))
        acts = torch.cat(acts).reshape(-1)
        ab, sb = t.class_bytes(0, classes)
        buf = torch.zeros(ab + sb, dtype=torch.uint8, device="cuda")
        buf[:ab] = acts
        torch.cuda.synchronize()
        t.import_classes(0, classes, buf)
        for n in sizes:
            x = torch.randint(0, 256, (n, row), generator=g, device="cuda", dtype=torch.uint8)
            x |= torch.randint(0, 256, (n, row), generator=g, device="cuda", dtype=torch.uint8)
            want = _want(acts, x, classes, clauses, n, bits, tol)
            # the first class of the largest sum
            cls = (want == want.max(1, keepdim=True).values).int().argmax(1)
            torch.cuda.synchronize()  # predict runs on the machine's own stream
            got = t.predict(x.reshape(-1), n)
            assert (t.stats()["predict_gemm"] == 0) == (lists is True)
            assert torch.equal(torch.as_tensor(got).cuda().reshape(-1).long(), cls), n
            sc = t.predict_scores(x.cpu().numpy().reshape(-1), n)
            assert np.array_equal(np.asarray(sc).reshape(n, classes), want.cpu().numpy()), n
        # few samples: every action word for the first request, lists after it
        for n in (3, 32, 1):
            x = torch.randint(0, 256, (n, row), generator=g, device="cuda", dtype=torch.uint8)
            want = _want(acts, x, classes, clauses, n, bits, tol).cpu().numpy()
            for _ in range(2):
                sc = t.predict_scores(x.cpu().numpy().reshape(-1), n)
                assert np.array_equal(np.asarray(sc).reshape(n, classes), want), n
    t.destroy()


def test_few_samples_then_lists(tm):
    """64 MB of actions: the second small request of a state makes the lists, a
    new state starts over."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    classes, features, clauses, tol = 8, 8192, 4096, 24
    row = features // 4
    t = tm.create("encoder", dict(hidden=classes, visible=features, clauses=clauses,
                                  clause_tolerance=tol, clause_maximum=64, specificity=9.0,
                                  reusable=False))
    t.stats_enable(True)
    ab, sb = t.class_bytes(0, classes)
    for again in range(2):
        buf = torch.zeros(ab + sb, dtype=torch.uint8, device="cuda")
        hit = torch.randint(0, ab, (classes * clauses * 40,), generator=g, device="cuda")
        buf[hit] = 1 << (again + 2)
        torch.cuda.synchronize()
        t.import_classes(0, classes, buf)
        for n in (5, 5, 32, 3):
            x = torch.randint(0, 256, (n, row), generator=g, device="cuda", dtype=torch.uint8)
            want = _want(buf[:ab], x, classes, clauses, n, 2 * features, tol).cpu().numpy()
            torch.cuda.synchronize()
            sc = t.predict_scores(x.cpu().numpy().reshape(-1), n)
            assert np.array_equal(np.asarray(sc).reshape(n, classes), want), n
    t.destroy()
