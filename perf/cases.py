"""What a user of this library has it do, as cases to time.

Each case is one call (or the few calls of one program run) through the public
Python entry points, over the workload families of bench.py: Gaussian-mixture
vectors under L2 and angle, words under edit distance, 2-D hotspot points under
L1, and update streams.  A case's "kind" says which calls are made:

  knn        Index.knn_device: ids in device memory, answers left there
  knn_host   Index.knn: ids and answers in host memory
  range      Index.range_device
  range_host Index.range
  range_ids  Index.range_ids (the hits themselves, not only their number)
  knn_rows   Index.knn_rows: queries given as vectors that are not in the index
  stream     index built, then Index.update_run over a stream of operations
  oneshot    index built, prepared for the form, one kNN batch answered: what
             one run of the command line does after it has read its files

Index construction belongs to prepare() where a serving program builds once and
asks many times, and to run() where the program is over after one batch.
Nothing here depends on how the library works inside.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import gts_b200 as gts
from gts_b200 import datagen

FORMS = {"plain": gts.FORM_PLAIN, "fast": gts.FORM_FAST}
METRICS = {"l1": 1, "l2": 2, "angle": 5, "edit": 6}
WORD_BYTES = 13          # a word of the generator below and its length, on average
DEV = "cuda"


# ---------------------------------------------------------------- the cases

def listed() -> list:
    return [
        # The headline: a serving loop that keeps ids and answers in device
        # memory and asks 10,000 queries at a time.
        dict(name="knn-l2-1m-k8", kind="knn", metric="l2", form="fast", n=1_000_000, dim=128, comps=256,
             sigma=0.2, q=10_000, k=8, ids=False),
        # The same data asked for long result lists, with the ids (one batch of
        # the mixed-k workload is about 2,500 queries).
        dict(name="knn-l2-1m-k64-ids", kind="knn", metric="l2", form="fast", n=1_000_000, dim=128, comps=256,
             sigma=0.2, q=2_500, k=64, ids=True),
        # Selectivity estimation: how many objects lie within the radius.
        dict(name="range-l2-1m", kind="range", metric="l2", form="fast", n=1_000_000, dim=128, comps=256,
             sigma=0.2, q=10_000, frac=0.001),
        # Interactive lookup: one query, host to host, ragged sizes.
        dict(name="knn-l2-50k-q1", kind="knn_host", metric="l2", form="fast", n=50_021, dim=300, comps=64,
             sigma=0.3, q=1, k=8, ids=True),
        # The library's default form (tree traversal) at the size of the headline.
        dict(name="knn-l2-1m-plain", kind="knn_host", metric="l2", form="plain", n=1_000_000, dim=128, comps=256,
             sigma=0.2, q=1_000, k=8, ids=True),
        # Near-duplicate listing: every hit of a radius, with ids and distances.
        dict(name="range-ids-l2-50k", kind="range_ids", metric="l2", form="plain", n=50_000, dim=300, comps=64,
             sigma=0.3, q=1_000, frac=0.001),
        # Spell checking: how many words lie within two edits.
        dict(name="range-edit-1m-r2", kind="range_host", metric="edit", form="plain", n=1_000_000, q=10_000, r=2),
        # One run of the command line over a word list: build, then nearest words.
        dict(name="oneshot-edit-200k", kind="oneshot", metric="edit", form="plain", n=200_000, q=1_000, k=16,
             ids=True),
        # Location data: very many cheap queries over very many small objects.
        dict(name="range-l1-10m", kind="range_host", metric="l1", form="plain", n=10_000_000, q=100_000,
             frac=0.0001),
        # Embeddings compared by angle; the queries are new vectors.
        dict(name="knn-rows-angle-100k", kind="knn_rows", metric="angle", form="plain", n=100_003, dim=300, comps=333,
             sigma=0.4, q=500, k=10, ids=True),
        # A stream of inserts, deletes and range queries over a fresh index.
        dict(name="stream-l2-100k", kind="stream", metric="l2", form="plain", n=100_000, dim=300, comps=64,
             sigma=0.3, ops=20_000, frac=0.001),
        # One run of the command line over vectors with the fast form: build,
        # prepare, one batch.
        dict(name="oneshot-l2-1m", kind="oneshot", metric="l2", form="fast", n=1_000_000, dim=128, comps=256,
             sigma=0.2, q=1_000, k=8, ids=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["knn", "knn", "range", "knn_host", "plain", "range_ids", "edit", "edit_oneshot", "l1",
                       "angle", "stream", "oneshot"])
    mix = dict(metric="l2", dim=rng.choice([24, 33, 64, 100, 128, 128, 200, 300]), comps=rng.randint(32, 256),
               sigma=round(rng.uniform(0.2, 0.3), 3))
    if kind == "knn":
        return dict(kind="knn", form="fast", n=_log_int(rng, 20_000, 1_000_000), q=_log_int(rng, 50, 10_000),
                    k=_log_int(rng, 1, 64), ids=rng.random() < 0.5, **mix)
    if kind == "range":
        return dict(kind="range", form="fast", n=_log_int(rng, 20_000, 1_000_000), q=_log_int(rng, 50, 10_000),
                    frac=round(math.exp(rng.uniform(math.log(2e-4), math.log(1e-3))), 6), **mix)
    if kind == "knn_host":
        return dict(kind="knn_host", form="fast", n=_log_int(rng, 5_000, 200_000), q=_log_int(rng, 1, 100),
                    k=_log_int(rng, 1, 32), ids=True, **mix)
    if kind == "plain":
        return dict(kind="knn_host", form="plain", n=_log_int(rng, 20_000, 1_000_000), q=_log_int(rng, 20, 1_000),
                    k=_log_int(rng, 1, 64), ids=rng.random() < 0.5, **mix)
    if kind == "range_ids":
        return dict(kind="range_ids", form="plain", n=_log_int(rng, 5_000, 100_000), q=_log_int(rng, 50, 1_000),
                    frac=round(math.exp(rng.uniform(math.log(2e-4), math.log(1e-3))), 6), **mix)
    if kind == "edit":
        return dict(kind="range_host", metric="edit", form="plain", n=_log_int(rng, 50_000, 1_000_000),
                    q=_log_int(rng, 100, 5_000), r=rng.randint(1, 3))
    if kind == "edit_oneshot":
        return dict(kind="oneshot", metric="edit", form="plain", n=_log_int(rng, 20_000, 200_000),
                    q=_log_int(rng, 20, 1_000), k=_log_int(rng, 1, 32), ids=True)
    if kind == "l1":
        return dict(kind="range_host", metric="l1", form="plain", n=_log_int(rng, 500_000, 10_000_000),
                    q=_log_int(rng, 1_000, 100_000), frac=0.0001)
    if kind == "angle":
        return dict(kind="knn_rows", metric="angle", form="plain", n=_log_int(rng, 5_000, 100_000),
                    dim=rng.choice([25, 64, 100, 300]), comps=rng.randint(16, 333), sigma=0.4,
                    q=_log_int(rng, 10, 500), k=_log_int(rng, 1, 32), ids=True)
    if kind == "stream":
        return dict(kind="stream", form="plain", n=_log_int(rng, 5_000, 100_000), ops=_log_int(rng, 1_000, 20_000),
                    frac=0.001, **mix)
    return dict(kind="oneshot", form="fast", n=_log_int(rng, 20_000, 500_000), q=_log_int(rng, 50, 1_000),
                k=_log_int(rng, 1, 32), ids=True, **mix)


# ---------------------------------------------------------------- inputs

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _mixture(n, case, g, centres=None):
    """Rows of the Gaussian mixture (centres ~ N(0, 1)); angle data are shifted
    off the origin as the tests' are."""
    dim = case["dim"]
    if centres is None:
        centres = torch.randn(case["comps"], dim, generator=g, device=DEV)
    comp = torch.randint(case["comps"], (n,), generator=g, device=DEV)
    rows = torch.randn(n, dim, generator=g, device=DEV).mul_(case["sigma"]).add_(centres[comp])
    if case["metric"] == "angle":
        rows += 0.5
    return rows, centres


def _hotspots(n, g, n_hot=500, sigma=0.005):
    """70 % of the points in Gaussian hotspots, the rest uniform."""
    hot = torch.rand(n_hot, 2, generator=g, device=DEV, dtype=torch.float64)
    pts = torch.rand(n, 2, generator=g, device=DEV, dtype=torch.float64)
    at = hot[torch.randint(n_hot, (n,), generator=g, device=DEV)]
    at += sigma * torch.randn(n, 2, generator=g, device=DEV, dtype=torch.float64)
    in_hot = torch.rand(n, 1, generator=g, device=DEV) < 0.7
    return torch.where(in_hot, at, pts).float()


def _words(n, g, median=8.0, max_len=34):
    """Lowercase words in host memory: log-normal lengths, Zipf(1.1) letters."""
    lens = torch.exp(math.log(median) + 0.5 * torch.randn(n, generator=g, device=DEV)).round().clamp(1, max_len).int()
    p = torch.arange(1, 27, device=DEV, dtype=torch.float64) ** -1.1
    cum = torch.cumsum(p / p.sum(), 0).float()
    letter = torch.searchsorted(cum, torch.rand(n, max_len, generator=g, device=DEV)).clamp(max=25)
    letter = letter.to(torch.uint8) + ord("a")
    letter[torch.arange(max_len, device=DEV)[None, :] >= lens[:, None]] = 0
    strs = torch.zeros(n, datagen.STR_STRIDE, dtype=torch.uint8, device=DEV)
    strs[:, :max_len] = letter
    return strs.cpu().numpy(), lens.cpu().numpy()


def _distances(case, a, b):
    """Distances of a's rows to b's, in 64 bits, pair by pair."""
    a, b = a.double(), b.double()
    if case["metric"] == "l1":
        return (a - b).abs().sum(-1)
    if case["metric"] == "l2":
        return (a - b).square().sum(-1).sqrt()
    cos = (a * b).sum(-1) / (a.norm(dim=-1) * b.norm(dim=-1))
    return torch.acos(cos.clamp(max=1.0)) * 180 / 3.1415926   # the metric's own constant


def _radius(case, rows, g):
    """The distance quantile of a sample of pairs, as bench.py picks radii."""
    i = torch.randint(len(rows), (2, 1_000_000 if rows.shape[1] <= 8 else 100_000), generator=g, device=DEV)
    d = _distances(case, rows[i[0]], rows[i[1]])
    kth = max(1, int(round(case["frac"] * len(d))))
    return float(torch.kthvalue(d, kth).values.float())


def _tree_height(n):
    """Levels that leave at most max_size (20) objects in a leaf at order 10."""
    h = 2
    while n / 10 ** (h - 1) > 20:
        h += 1
    return h


def _inputs(case, seed):
    """Everything that is random in a case: from the seed alone."""
    g = _gen(seed)
    n, x = case["n"], {}
    if case["metric"] == "edit":
        x["words"] = _words(n, g)
    elif case["metric"] == "l1":
        x["rows"] = _hotspots(n, g)
    else:
        x["rows"], centres = _mixture(n, case, g)
        if case["kind"] == "knn_rows":
            x["queries"] = _mixture(case["q"], case, g, centres)[0]
    if "frac" in case:
        x["r"] = _radius(case, x["rows"], g)
    elif "r" in case:
        x["r"] = float(case["r"])
    if "q" in case:
        x["qids"] = torch.randperm(n, generator=g, device=DEV)[:case["q"]].int()
    if case["kind"] == "stream":
        x["flags"], x["ids"] = datagen.update_stream(n, case["ops"], int(seed) % (1 << 31))
    return x


def _hit_room(case):
    return 4 * int(case["q"] * (1 + case["frac"] * case["n"]))


def _build(case, x):
    stream = torch.cuda.current_stream().cuda_stream
    h = _tree_height(case["n"])
    if case["metric"] == "edit":
        return gts.Index(None, 6, strs=x["words"][0], lens=x["words"][1], max_h=h)
    rows = x["rows"]
    return gts.Index.from_device(rows.data_ptr(), rows.shape[0], rows.shape[1], METRICS[case["metric"]],
                                 stream=stream, max_h=h)


def prepare(case, seed):
    x = _inputs(case, seed)
    s = {"case": case, **{key: x[key] for key in ("r", "flags", "ids") if key in x}}
    kind, form = case["kind"], FORMS[case["form"]]
    if kind in ("stream", "oneshot"):   # the program builds its index itself
        s["x"] = x
        if "qids" in x:
            s["qids"] = x["qids"].cpu().numpy()
        return s
    s["idx"] = _build(case, x)
    s["idx"].prepare(form, torch.cuda.current_stream().cuda_stream)
    if kind == "knn_rows":
        s["queries"] = x["queries"].cpu().numpy()
        return s
    if kind in ("knn", "range"):
        q, k = case["q"], case.get("k", 1)
        s["qids"] = x["qids"]
        if kind == "range":
            s["counts"] = torch.empty(q, dtype=torch.int32, device=DEV)
        else:
            s["kth"] = torch.empty(q, dtype=torch.float32, device=DEV)
            if case["ids"]:
                s["nn"] = torch.empty(q, k, dtype=torch.int32, device=DEV)
                s["dists"] = torch.empty(q, k, dtype=torch.float32, device=DEV)
    else:
        s["qids"] = x["qids"].cpu().numpy()
    if kind == "range_ids":   # room for the hits, as a program that keeps its buffers has
        s["hit_ids"] = np.full(_hit_room(case), -1, np.int32)
        s["hit_dists"] = np.zeros(_hit_room(case), np.float32)
    if kind != "range_ids" and case["q"] >= 2000:
        # a serving program has asked this index for batches like this one
        # before: whatever the library settles in the first of them is settled
        other = torch.randint(case["n"], (case["q"],), generator=_gen(seed + 1), device=DEV).int()
        run({**s, "qids": other if kind in ("knn", "range") else other.cpu().numpy()})
    return s


# ---------------------------------------------------------------- one pass

def run(s):
    case = s["case"]
    kind, form = case["kind"], FORMS[case["form"]]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "knn":
        ids, dists = s.get("nn"), s.get("dists")
        s["idx"].knn_device(s["qids"].data_ptr(), case["q"], case["k"], s["kth"].data_ptr(),
                            ids.data_ptr() if ids is not None else 0,
                            dists.data_ptr() if dists is not None else 0, form=form, stream=stream)
        return {"kth": s["kth"], "ids": ids, "dists": dists}
    if kind == "knn_host":
        return _named(s["idx"].knn(s["qids"], case["k"], form=form, return_ids=case["ids"]))
    if kind == "range":
        s["idx"].range_device(s["qids"].data_ptr(), case["q"], s["r"], s["counts"].data_ptr(), stream=stream,
                              form=form)
        return {"counts": s["counts"]}
    if kind == "range_host":
        return {"counts": s["idx"].range(s["qids"], s["r"], form=form)}
    if kind == "range_ids":
        counts, offsets, ids, dists = s["idx"].range_ids(s["qids"], s["r"])
        s["hit_ids"][:len(ids)] = ids
        s["hit_dists"][:len(dists)] = dists
        return {"counts": counts, "offsets": offsets, "ids": s["hit_ids"], "dists": s["hit_dists"]}
    if kind == "knn_rows":
        return _named(s["idx"].knn_rows(s["queries"], case["k"], return_ids=case["ids"]))
    with _build(case, s["x"]) as idx:
        if kind == "stream":
            counts, _, _ = idx.update_run(s["flags"], s["ids"], s["r"])
            answers = np.full(case["ops"], -1, np.int32)   # by operation
            answers[s["flags"] == 2] = counts
            tree = idx.export()["id_list"]                 # the tree that the stream leaves
            order = np.full(case["n"] + case["ops"], -1, np.int32)
            order[:len(tree)] = tree
            return {"answers": answers, "order": order}
        idx.prepare(form, stream)
        return _named(idx.knn(s["qids"], case["k"], form=form, return_ids=case["ids"]))


def _named(got):
    kth, ids, dists = got if isinstance(got, tuple) else (got, None, None)
    return {"kth": kth, "ids": ids, "dists": dists}


# ---------------------------------------------------------------- what it comes to

def work(case) -> dict:
    """What a pass cannot do without.  A kNN answer needs its query and its k
    objects read, a range answer its hits (an object shared by several queries
    once); a program that builds needs every object read and its tree-ordered
    copy written."""
    n, q, k = case["n"], case.get("q", 0), case.get("k", 1)
    row = WORD_BYTES if case["metric"] == "edit" else 4 * case.get("dim", 2)
    per_pair = 17 * 9 if case["metric"] == "edit" else 3 * case.get("dim", 2)
    if case["kind"] == "stream":
        q = case["ops"] // 10
    hits = q * k if "k" in case else q * case["frac"] * n if "frac" in case else q
    b = 4 * q + q * row + min(n, hits) * row + 4 * q
    f = hits * per_pair
    if case.get("ids"):
        b += 8 * q * k
    if case["kind"] == "range_ids":
        b += 8 * hits + 4 * q
    if case["kind"] in ("stream", "oneshot"):
        b += 2 * n * row + 8 * n
        f += (_tree_height(n) - 1) * n * per_pair
        if case["kind"] == "stream":   # and the tree that the stream leaves
            b += 2 * n * row + 8 * n + 8 * case["ops"]
            f += (_tree_height(n) - 1) * n * per_pair
    return {"bytes": float(b), "flops": float(f)}


def exact(case, seed):
    """The distances in 64 bits; counts and ids are whole numbers."""
    if case["metric"] == "edit" or case["kind"] in ("range", "range_host", "stream"):
        return None
    x = _inputs(case, seed)
    rows = x["rows"].double()
    by_id = case["kind"] != "knn_rows"
    qids = x["qids"].long()
    queries = rows[qids] if by_id else x["queries"].double()
    out, hits = [], []
    if case["metric"] == "angle":
        unit = rows / rows.norm(dim=1, keepdim=True)
    else:
        sq = rows.square().sum(1)
    for i in range(0, case["q"], 128):
        qs = queries[i:i + 128]
        # 64-bit products pick the objects; their distances are then made pair by pair
        if case["metric"] == "angle":
            near = -(qs @ unit.T)
        else:
            near = sq[None, :] - 2 * (qs @ rows.T)
        if case["kind"] == "range_ids":
            near += qs.square().sum(1)[:, None]
            for j in range(len(qs)):
                at = torch.nonzero(near[j] <= (x["r"] * 1.001) ** 2)[:, 0]
                d = _distances(case, rows[at], qs[j][None, :])
                d[at == qids[i + j]] = 0.0
                hits.append(d[d.float() <= x["r"]].sort().values)
            continue
        at = torch.topk(near, min(case["k"] + 8, case["n"]), dim=1, largest=False).indices
        d = _distances(case, rows[at], qs[:, None, :])
        if by_id:
            d[at == qids[i:i + 128, None]] = 0.0
        out.append(d.sort(dim=1).values[:, :case["k"]])
    if case["kind"] == "range_ids":
        dists = torch.zeros(_hit_room(case), dtype=torch.float64, device=DEV)
        hits = torch.cat(hits)
        dists[:len(hits)] = hits
        return {"counts": None, "offsets": None, "ids": None, "dists": dists}
    out = torch.cat(out)
    return {"kth": out[:, -1], "ids": None, "dists": out if case.get("ids") else None}
