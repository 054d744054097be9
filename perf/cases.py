"""Performance cases of the Tsetlin-machine framework: the calls its users make,
over the sizes they make them at, through the package's public entry points.

    listed()           named cases
    draw(rng)          one more case of the same ranges
    prepare(case, s)   inputs (from seed s), machines and buffers a program holds
    run(state)         one pass; returns its outputs
    work(case)         bytes and operations one pass cannot do without
    exact(case, s)     what run() returns, in 64 bits, where outputs are fractions

Kinds of case:
  predict  classes or codes of n samples from a resident machine, inputs and
           outputs in host memory (a request) or on the GPU (an evaluation)
  train    one train call of a machine from its inputs to its final automata
  search   one device-resident round of the hyper-parameter search
  pack     set-bit lists to flip-interleaved sample rows
  score    the evaluator's metrics of predictions against the truth
"""
import math
import os
import random
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "lua-santoku-tsetlin_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import santoku_tsetlin as tm  # noqa: E402

DEV = "cuda"


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # an interactive request: one sample against the plain classifier
        dict(name="predict-one-plain", kind="predict", type="classifier", data="prototype",
             classes=10, features=784, clauses=256, n=1, host=True),
        # a small request against a machine whose actions (168 MB) exceed L2
        dict(name="predict-few-sparse", kind="predict", type="classifier", data="sparse",
             classes=20, features=16384, clauses=2048, n=5, host=True),
        # the plain classifier's test set, from host memory
        dict(name="predict-set-plain", kind="predict", type="classifier", data="prototype",
             classes=10, features=784, clauses=256, n=2000, host=True),
        # the large sparse classifier's test set
        dict(name="predict-set-sparse", kind="predict", type="classifier", data="sparse",
             classes=20, features=16384, clauses=2048, n=20000, host=False),
        # the encoder's holdout
        dict(name="predict-set-encoder", kind="predict", type="encoder", data="latent",
             classes=256, features=4096, clauses=1024, n=20000, host=False),
        # the plain classifier's whole training
        dict(name="train-plain", kind="train", type="classifier", data="prototype", classes=10,
             features=784, clauses=256, n=8000, epochs=10, target=50.0, specificity=10.0,
             state=8, include_bits=1, ind=False, host=True),
        # the large sparse classifier on a share of its samples (1,024-word rows)
        dict(name="train-sparse", kind="train", type="classifier", data="sparse", classes=20,
             features=16384, clauses=2048, n=6000, epochs=2, target=200.0, specificity=25.0,
             state=8, include_bits=1, ind=False, host=False),
        # the encoder on a share of its samples (256-word rows, every sample
        # trains every unit)
        dict(name="train-encoder", kind="train", type="encoder", data="latent", classes=256,
             features=4096, clauses=1024, n=1024, epochs=1, target=100.0, specificity=15.0,
             state=8, include_bits=1, ind=False, host=False),
        # an individualized encoder: every hidden bit has its own, odd, feature
        # count; two include bits
        dict(name="train-ragged", kind="train", type="encoder", data="latent", classes=37,
             features=693, clauses=72, n=1999, epochs=3, target=40.0, specificity=12.0,
             state=8, include_bits=2, ind=True, host=False),
        # a round of the hyper-parameter search: uneven machines trained
        # together, scored after every epoch
        dict(name="search-round", kind="search", machines=16, classes=10, features=784,
             n=6000, n_test=1500, epochs=3, patience=2),
        # packing the sparse classifier's inputs (1.5 % set bits)
        dict(name="pack-sparse", kind="pack", n=20000, features=16384, density=0.015, flip=True),
        # Hamming scores of the encoder's holdout codes
        dict(name="score-codes", kind="score", type="encoder", classes=256, n=20000),
    ]


def _logu(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# word tests (clauses x samples x row words) the largest listed predict and
# train cases make; drawn cases stay below
_MOST_PREDICT = 256 * 1024 * 20000 * 256
_MOST_TRAIN = 256 * 1024 * 1024 * 256 // 2


def draw(rng):
    pick = rng.random()
    if pick < 0.40:
        enc = rng.random() < 0.3
        c = dict(kind="predict", type="encoder" if enc else "classifier",
                 data="latent" if enc else rng.choice(["prototype", "sparse"]),
                 classes=_logu(rng, 8, 256) if enc else _logu(rng, 2, 40),
                 features=_logu(rng, 64, 16384), clauses=_logu(rng, 2, 256) * 8,
                 n=_logu(rng, 1, 20000), host=rng.random() < 0.5)
        if c["n"] > 4096:
            c["host"] = False
        while c["classes"] * c["clauses"] * (c["features"] // 16) > 256 * 1024 * 256:
            c["clauses"] = max(8, c["clauses"] // 16 * 8)
        while c["classes"] * c["clauses"] * (c["features"] // 16) * c["n"] > _MOST_PREDICT:
            c["n"] = c["n"] // 2 + 1
        return c
    if pick < 0.78:
        enc = rng.random() < 0.35
        ind = rng.random() < 0.25
        c = dict(kind="train", type="encoder" if enc else "classifier",
                 data="latent" if enc else rng.choice(["prototype", "sparse"]),
                 classes=_logu(rng, 8, 128) if enc else _logu(rng, 2, 24),
                 features=_logu(rng, 64, 2048 if ind else 16384),
                 clauses=_logu(rng, 2, 128) * 8, n=_logu(rng, 200, 10000),
                 epochs=rng.randint(1, 6), target=float(_logu(rng, 20, 400)),
                 specificity=float(round(rng.uniform(2.0, 40.0), 2)),
                 state=rng.choice([8, 8, 8, 8, 8, 6, 10]), include_bits=rng.choice([1, 1, 1, 2, 3]),
                 ind=ind, host=(not ind) and rng.random() < 0.4)

        def cost():
            act = 1.0 if c["type"] == "encoder" else min(1.0, 2.0 / c["classes"])
            return (c["classes"] * c["clauses"] * (c["features"] / 16.0 + 40) * c["n"] *
                    c["epochs"] * act)
        while cost() > _MOST_TRAIN / 4:
            if c["epochs"] > 1:
                c["epochs"] -= 1
            elif c["n"] > 400:
                c["n"] = c["n"] * 2 // 3 + 1
            else:
                c["clauses"] = max(8, c["clauses"] // 16 * 8)
        return c
    if pick < 0.84:
        return dict(kind="search", machines=rng.randint(3, 16), classes=rng.randint(3, 16),
                    features=2 * _logu(rng, 100, 500), n=_logu(rng, 500, 4000),
                    n_test=_logu(rng, 200, 1500), epochs=rng.randint(1, 3),
                    patience=rng.randint(0, 2))
    if pick < 0.92:
        c = dict(kind="pack", n=_logu(rng, 50, 20000), features=_logu(rng, 64, 16384),
                 density=round(rng.uniform(0.005, 0.3), 3), flip=rng.random() < 0.8)
        while c["n"] * c["features"] > 20000 * 16384 // 2:
            c["n"] = c["n"] // 2 + 1
        return c
    enc = rng.random() < 0.5
    return dict(kind="score", type="encoder" if enc else "classifier",
                classes=_logu(rng, 8, 256) if enc else _logu(rng, 2, 100),
                n=_logu(rng, 500, 100000 if not enc else 40000))


# ---------------------------------------------------------------------------
# inputs, from the seed, with the distributions of the benchmark's workloads
# ---------------------------------------------------------------------------
def _gen(seed, salt):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 1000003 + salt) & 0x7FFFFFFF)
    return g


def _pack(bits):
    """bool (n, B) -> uint8 (n, ceil(B / 8)), LSB first."""
    n, b = bits.shape
    nb = (b + 7) // 8
    if b % 8:
        bits = torch.nn.functional.pad(bits, (0, 8 * nb - b))
    w = torch.tensor([1, 2, 4, 8, 16, 32, 64, 128], device=bits.device, dtype=torch.uint8)
    return (bits.view(n, nb, 8).to(torch.uint8) * w).sum(dim=2, dtype=torch.uint8)


def _flip_pack(bits):
    return _pack(torch.cat([bits, ~bits], dim=1))


def _sparse_probs(features, classes, density=0.015, zipf=1.1, boost=8.0):
    """Zipf activation probabilities with `density` mean, a boosted feature
    subset per class (the same for every seed)."""
    r = np.random.default_rng(104730 + features)
    rank = r.permutation(features)
    base = 1.0 / np.power(rank + 1.0, zipf)
    lo, hi = 0.0, 1.0 / base.min()
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        if np.minimum(base * mid, 1.0).mean() < density:
            lo = mid
        else:
            hi = mid
    p = np.repeat(np.minimum(base * hi, 1.0)[None, :], classes, axis=0)
    for c in range(classes):
        pick = r.choice(features, size=min(features, max(4, features // 82)), replace=False)
        p[c, pick] = np.minimum(p[c, pick] * boost, 1.0)
    return torch.tensor(p, dtype=torch.float32, device=DEV)


class _Source:
    """Feature bits and truth of a workload, in chunks of samples."""

    def __init__(self, case, seed, flip=0.1):
        self.data, self.features, self.classes = case["data"], case["features"], case["classes"]
        self.g = _gen(seed, 1)
        self.flip = flip
        p = torch.Generator(device=DEV)
        p.manual_seed(7919 + self.features)
        if self.data == "prototype":
            self.protos = torch.rand(self.classes, self.features, generator=p, device=DEV) < 0.2
        elif self.data == "sparse":
            self.probs = _sparse_probs(self.features, self.classes)
        else:
            self.px = torch.randn(64, self.features, generator=p, device=DEV)
            self.pc = torch.randn(64, self.classes, generator=p, device=DEV)

    def take(self, m):
        """(bits (m, features), truth): truth is int64 classes, or bool codes."""
        if self.data == "latent":
            z = torch.randn(m, 64, generator=self.g, device=DEV)
            bits = (z @ self.px) > 0
            bits ^= torch.rand(m, self.features, generator=self.g, device=DEV) < 0.05
            return bits, (z @ self.pc) > 0
        y = torch.randint(self.classes, (m,), generator=self.g, device=DEV)
        u = torch.rand(m, self.features, generator=self.g, device=DEV)
        if self.data == "prototype":
            return self.protos[y] ^ (u < self.flip), y
        return u < self.probs[y], y


def _dense_rows(case, seed, n, flip=0.1, negated=True):
    src = _Source(case, seed, flip)
    xs, ys = [], []
    for i in range(0, n, 4096):
        bits, y = src.take(min(4096, n - i))
        xs.append(_flip_pack(bits) if negated else _pack(bits))
        ys.append(y if y.dtype == torch.int64 else _pack(y))
    return torch.cat(xs).reshape(-1), torch.cat(ys).reshape(-1)


def _trained_actions(case, seed, machine):
    """Action bytes as training leaves them: each clause includes about 32
    literals that one sample of its class satisfies."""
    src = _Source(case, seed ^ 0x5A5A)
    g = _gen(seed, 2)
    lits = 2 * case["features"]
    clauses = machine.info()["clauses"]
    total = case["classes"] * clauses
    out = []
    for i in range(0, total, 4096):
        m = min(4096, total - i)
        bits, _ = src.take(m)
        row = torch.cat([bits, ~bits], dim=1)
        at = torch.randint(lits, (m, 64), generator=g, device=DEV)
        keep = torch.zeros(m, lits, dtype=torch.bool, device=DEV)
        keep.scatter_(1, at, True)
        out.append(_pack(row & keep))
    return torch.cat(out).reshape(-1)


def _import_actions(machine, acts, classes):
    a, s = machine.class_bytes(0, classes)
    buf = torch.zeros(a + s, dtype=torch.uint8, device=DEV)
    buf[:a] = acts
    torch.cuda.synchronize()
    machine.import_classes(0, classes, buf)


def _create(case, seed, reusable=True, **extra):
    enc = case["type"] == "encoder"
    t = dict(clauses=case["clauses"], clause_tolerance=64, clause_maximum=64,
             specificity=case.get("specificity", 10.0), target=case.get("target", 50.0),
             state=case.get("state", 8), include_bits=case.get("include_bits", 1),
             reusable=reusable, seed=int(seed) & 0xFFFFFFFF)
    if enc:
        t.update(visible=case["features"], hidden=case["classes"])
    else:
        t.update(features=case["features"], classes=case["classes"])
    t.update(extra)
    return tm.create(case["type"], t)


def _ind_sizes(case):
    """Feature count of every class of an individualized machine."""
    r = random.Random(case["features"] * 131 + case["classes"])
    lo = max(1, case["features"] // 8)
    return [r.randint(lo, case["features"]) for _ in range(case["classes"])]


def _ind_rows(case, seed, n):
    """Individualized rows: class h sees the first k_h of the features."""
    src = _Source(case, seed)
    bits, y = src.take(n)
    blocks, off = [], [0]
    for k in _ind_sizes(case):
        b = _flip_pack(bits[:, :k]).reshape(-1)
        blocks.append(b)
        off.append(off[-1] + b.numel())
    y = y if y.dtype == torch.int64 else _pack(y).reshape(-1)
    return torch.cat(blocks), np.array(off, dtype=np.int64), y


def _search_params(case, seed):
    r = np.random.default_rng(case["machines"] * 7 + case["features"])
    out = []
    for i in range(case["machines"]):
        clauses = max(8, int(round(math.exp(r.uniform(math.log(64), math.log(4096))) / 8.0)) * 8)
        out.append(dict(negated=bool(r.random() < 0.5), clauses=clauses,
                        specificity=float(r.uniform(2.0, 40.0)),
                        target=float(int(r.uniform(20.0, 400.0))), seed=int(seed) * 97 + i))
    return out


def prepare(case, seed):
    k = case["kind"]
    s = dict(case=case)
    if k == "predict":
        s["m"] = _create(case, seed, reusable=False)
        _import_actions(s["m"], _trained_actions(case, seed, s["m"]), case["classes"])
        x, _ = _dense_rows(case, seed, case["n"])
        s["x"] = x.cpu().numpy() if case["host"] else x
    elif k == "train":
        extra = {}
        tbl = dict(samples=case["n"], iterations=case["epochs"])
        if case["ind"]:
            extra["individualized"] = True
            extra["feat_offsets"] = np.concatenate([[0], np.cumsum(_ind_sizes(case))])
            x, off, y = _ind_rows(case, seed, case["n"])
            tbl["dim_offsets"] = off
        else:
            x, y = _dense_rows(case, seed, case["n"])
        if case["host"]:
            x, y = x.cpu().numpy(), y.cpu().numpy()
        enc = case["type"] == "encoder"
        tbl["sentences" if enc else "problems"] = x
        tbl["codes" if enc else "solutions"] = y
        s["m"] = _create(case, seed, **extra)
        s["tbl"] = tbl
        i = s["m"].info()
        if case["ind"]:
            s["ab"], s["sb"] = i["action_chunks"], i["state_chunks"]
        else:
            s["ab"], s["sb"] = s["m"].class_bytes(0, case["classes"])
            s["out"] = torch.empty(s["ab"] + s["sb"], dtype=torch.uint8, device=DEV)
    elif k == "search":
        base = dict(case, data="prototype")
        n, nt = case["n"], case["n_test"]
        s["ms"], s["tbls"], xs, rows = [], [], [], {}
        for p in _search_params(case, seed):
            neg = p["negated"]
            if neg not in rows:
                x, y = _dense_rows(base, seed, n + nt, flip=0.4, negated=neg)
                rows[neg] = (x, x.numel() // (n + nt), y)
            x, nb, y = rows[neg]
            f = case["features"] if neg else case["features"] // 2
            s["ms"].append(_create(dict(case, type="classifier", features=f, clauses=p["clauses"],
                                        specificity=p["specificity"], target=p["target"]),
                                   p["seed"]))
            s["tbls"].append(dict(samples=n, problems=x[:n * nb], solutions=y[:n],
                                  iterations=case["epochs"]))
            xs.append(x[n * nb:])
            truth = y[n:]
        s["test"] = dict(samples=nt, problems_each=[v.contiguous() for v in xs],
                         solutions=truth.contiguous())
        s["outs"] = [torch.empty(sum(m.class_bytes(0, case["classes"])), dtype=torch.uint8,
                                 device=DEV) for m in s["ms"]]
    elif k == "pack":
        g = _gen(seed, 3)
        n, f = case["n"], case["features"]
        step = max(1, (64 << 20) // f)
        idx = [torch.nonzero(torch.rand(min(step, n - i) * f, generator=g, device=DEV) <
                             case["density"]).reshape(-1) + i * f for i in range(0, n, step)]
        s["bits"] = torch.cat(idx)
    else:
        g = _gen(seed, 4)
        n, c = case["n"], case["classes"]
        if case["type"] == "encoder":
            truth = torch.rand(n, c, generator=g, device=DEV) < 0.5
            wrong = torch.rand(n, c, generator=g, device=DEV) < torch.rand(
                c, generator=g, device=DEV) * 0.3
            s["truth"], s["pred"] = _pack(truth).reshape(-1), _pack(truth ^ wrong).reshape(-1)
        else:
            s["truth"] = torch.randint(c, (n,), generator=g, device=DEV)
            other = torch.randint(c, (n,), generator=g, device=DEV)
            hit = torch.rand(n, generator=g, device=DEV) < 0.9
            s["pred"] = torch.where(hit, s["truth"], other)
    torch.cuda.synchronize()
    return s


def run(s):
    case = s["case"]
    k = case["kind"]
    if k == "predict":
        return s["m"].predict(s["x"], case["n"])
    if k == "train":
        s["m"].train(s["tbl"])
        if case["ind"]:
            return s["m"].export_state()
        return s["m"].export_classes(0, case["classes"], s["out"])
    if k == "search":
        r = tm.train_batch_search(s["ms"], s["tbls"], s["test"], patience=case["patience"])
        for m, o in zip(s["ms"], s["outs"]):
            m.export_classes(0, case["classes"], o)
        return [r["scores"], r["final"], r["best"], r["epochs"].astype(np.int64),
                r["best_epoch"].astype(np.int64)] + s["outs"]
    if k == "pack":
        return tm.bits_to_cvec(s["bits"], case["n"], case["features"], case["flip"])
    if case["type"] == "encoder":
        r = tm.encoding_accuracy(s["pred"], s["truth"], case["n"], case["classes"])
        return np.array([r["mean_hamming"], r["ber_min"], r["ber_max"], r["ber_std"]] + r["bits"])
    r = tm.class_accuracy(s["pred"], s["truth"], case["n"], case["classes"])
    per = [v for c in r["classes"] for v in (c["precision"], c["recall"], c["f1"])]
    return np.array([r["precision"], r["recall"], r["f1"]] + per)


# ---------------------------------------------------------------------------
# work and exact values
# ---------------------------------------------------------------------------
def _units(case):
    """[(row bytes, clauses, samples trained on average)] of a machine's classes."""
    sizes = _ind_sizes(case) if case.get("ind") else [case["features"]] * case["classes"]
    part = 1.0
    if case["type"] == "classifier":
        c = case["classes"]
        part = 1.0 / c + (1.0 - 1.0 / c) / c
    return [((2 * f + 7) // 8, (case["clauses"] + 7) // 8 * 8, part) for f in sizes]


def work(case):
    k = case["kind"]
    if k == "predict":
        row = (2 * case["features"] + 7) // 8
        m = case["classes"] * ((case["clauses"] + 7) // 8 * 8)
        out = 8 if case["type"] == "classifier" else (case["classes"] + 7) // 8
        return dict(bytes=m * row + case["n"] * (row + out), flops=2.0 * m * case["n"] * row * 8)
    if k == "train":
        by = fl = 0.0
        for row, clauses, part in _units(case):
            by += clauses * row * case.get("state", 8)
            fl += 2.0 * clauses * row * 8 * case["n"] * case["epochs"] * part
        rows = sum(u[0] for u in _units(case)) if case["ind"] else _units(case)[0][0]
        return dict(bytes=by + case["n"] * (rows + 8), flops=fl)
    if k == "search":
        by = fl = 0.0
        for p in _search_params(case, 0):
            f = case["features"] if p["negated"] else case["features"] // 2
            u = _units(dict(type="classifier", classes=case["classes"], features=f,
                            clauses=p["clauses"]))
            for row, clauses, part in u:
                by += clauses * row * 8
                fl += 2.0 * clauses * row * 8 * case["epochs"] * (
                    case["n"] * part + case["n_test"])
        by += (case["n"] + case["n_test"]) * 1.5 * (2 * case["features"] / 8.0)
        return dict(bytes=by, flops=fl)
    if k == "pack":
        row = ((2 if case["flip"] else 1) * case["features"] + 7) // 8
        return dict(bytes=case["n"] * (row + 8.0 * case["density"] * case["features"]), flops=0)
    per = 2 * ((case["classes"] + 7) // 8) if case["type"] == "encoder" else 16
    return dict(bytes=case["n"] * per, flops=0)


def exact(case, seed):
    """The metrics in double precision; every other output is whole numbers."""
    if case["kind"] != "score":
        return None
    s = prepare(case, seed)
    n, c = case["n"], case["classes"]
    if case["type"] == "encoder":
        d = (s["pred"] ^ s["truth"]).view(n, -1)
        bits = torch.stack([(d >> b) & 1 for b in range(8)], dim=2).reshape(n, -1)[:, :c]
        wrong = bits.to(torch.int64).sum(dim=0).cpu().numpy().astype(np.float64)
        ber = wrong / n
        mean = wrong.sum() / (float(n) * c)
        std = math.sqrt(((ber - mean) ** 2).sum() / (c - 1)) if c > 1 else 0.0
        return np.concatenate([[1 - mean, 1 - ber.min(), 1 - ber.max(), std], ber])
    t, p = s["truth"].cpu().numpy(), s["pred"].cpu().numpy()
    tp = np.bincount(t[t == p], minlength=c).astype(np.float64)
    fp = np.bincount(p[t != p], minlength=c).astype(np.float64)
    fn = np.bincount(t[t != p], minlength=c).astype(np.float64)
    with np.errstate(divide="ignore", invalid="ignore"):
        pr = np.where(tp + fp > 0, tp / (tp + fp), 0.0)
        re = np.where(tp + fn > 0, tp / (tp + fn), 0.0)
        f1 = np.where(pr + re > 0, 2 * pr * re / (pr + re), 0.0)
    return np.concatenate([[pr.mean(), re.mean(), f1.mean()], np.stack([pr, re, f1], 1).ravel()])
