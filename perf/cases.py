"""Timed workloads of the distance library, from one small call to the largest.

listed() names the cases; draw() gives others of the same ranges.  A case is a
dict of plain values; prepare() makes what a user's program has in hand before
the call (sketches resident on the device, a server, a captured batch, genomes
or reads), run() makes one pass through the public API, exact() recomputes the
result in 64 bits with torch alone, work() counts what a pass cannot do
without.

Sketches are bin-level: a tree over samples, along whose branches each 14-bit
bin value is inherited or, with probability 1 - (1 - c)^k (1 - a), drawn
anew (c ~ U(0, 0.03), a ~ U(0, 0.2) per branch), on a random recursive tree or
on clades of log-normal size under one root.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "pp-sketchlib_b200"))

from sketchlib_b200 import capi  # noqa: E402

BBITS = 14
DEVICE = "cuda:0"
EXACT_LIMIT = 2.0e12          # bin comparisons exact() takes on (about 10 s)


def _ctx() -> capi.Context:
    """The program's one context: kept for its lifetime, as its stream and
    scratch are."""
    if not hasattr(_ctx, "ctx"):
        torch.zeros(1, device=DEVICE)
        _ctx.ctx = capi.Context(0)
    return _ctx.ctx


# ------------------------------------------------------------------- cases

def _case(kind, **kw):
    c = dict(kind=kind, n=0, nq=0, k0=15, dk=2, K=8, s64=156, tree="random", random="none",
             out="core_acc", knn=0, length=0)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest all-vs-all in use: one lineage of 64 genomes
        _case("self", name="self_64", n=64),
        # a collection that fits one lab's study, an odd size, Jaccards per k with a
        # Monte Carlo random-match table, the reference's default k set
        _case("self", name="self_1003_table", n=1003, k0=13, dk=4, K=5, random="table",
              out="jaccard"),
        # the plain all-vs-all of the benchmark
        _case("self", name="self_4096", n=4096),
        # a species-wide collection in clades, equal-base random matches
        _case("self", name="self_16001_clades", n=16001, tree="clades", random="equal"),
        # new samples against a collection, all distances kept
        _case("query", name="query_300_20011", n=20011, nq=300, tree="clades"),
        # one isolate looked up in a resident collection: latency
        _case("query_knn", name="lookup_1_30011", n=30011, nq=1, K=10, tree="clades", knn=5),
        # a serving request of 100 queries (page-locked words in, neighbours out)
        _case("serve", name="serve_100_30011", n=30011, nq=100, K=10, tree="clades", knn=5),
        # host sketches in, host distances out in one call
        _case("host", name="host_3001", n=3001),
        # a neighbour graph of a collection
        _case("knn", name="knn_6007", n=6007, tree="clades", knn=10),
        # unrelated databases of different sizes, k sets and widths in one launch
        _case("batch", name="batch_12", n=12),
        # assemblies sketched on the device
        _case("sketch", name="sketch_64x2.5M", n=64, length=2_500_000),
        # read sets sketched from host memory with exact k-mer counts
        _case("reads", name="reads_4x20M", n=4, length=2_000_000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["self", "self", "self", "query", "query", "query_knn", "serve", "host",
                       "knn", "batch", "sketch", "reads"])
    K = rng.randint(4, 10)
    c = dict(K=K, k0=rng.choice([13, 15, 17]), dk=2 if K > 6 else rng.choice([2, 4]),
             s64=rng.choice([16, 64, 156, 157, 312]), tree=rng.choice(["random", "clades"]),
             random=rng.choice(["none", "none", "equal", "table"]))
    # keeps every drawn case below the largest listed one, whatever its width
    shrink = math.sqrt(min(1.0, 8 * 156 / (K * c["s64"])))
    if kind == "self":
        return _case(kind, n=_log_int(rng, 30, 11000 * shrink),
                     out=rng.choice(["core_acc", "core_acc", "jaccard", "counts"]), **c)
    if kind in ("query", "query_knn", "serve"):
        knn = 0 if kind == "query" else rng.randint(1, 20)
        return _case(kind, n=_log_int(rng, 500, 24000 * shrink ** 2), nq=_log_int(rng, 1, 1500),
                     knn=knn, **c)
    if kind == "host":
        return _case(kind, n=_log_int(rng, 100, 4000 * shrink ** 2),
                     nq=rng.choice([0, rng.randint(1, 400)]), **c)
    if kind == "knn":
        return _case(kind, n=_log_int(rng, 100, 8000 * shrink), knn=rng.randint(1, 50), **c)
    if kind == "batch":
        return _case(kind, n=rng.randint(2, 16))
    if kind == "sketch":
        return _case(kind, n=_log_int(rng, 1, 48), length=_log_int(rng, 30_000, 3_000_000),
                     K=K, k0=c["k0"], dk=c["dk"], s64=c["s64"])
    return _case(kind, n=rng.randint(1, 4), length=_log_int(rng, 200_000, 2_000_000),
                 K=K, k0=c["k0"], dk=c["dk"])


def _kmers(case):
    return [case["k0"] + case["dk"] * i for i in range(case["K"])]


# ------------------------------------------------------------------ inputs

def _tree(n, clades, rng):
    """Parents of n samples: a random recursive tree, or 200 clades (fewer for
    small n) of log-normal size under one root."""
    parent = np.full(n, -1, np.int64)
    if not clades:
        parent[1:] = (rng.random(n - 1) * np.arange(1, n)).astype(np.int64)
        return parent
    n_cl = max(1, min(200, (n - 1) // 8))
    w = rng.lognormal(0.0, 1.0, n_cl)
    first = 1 + np.floor(np.concatenate([[0], np.cumsum(w)[:-1]]) / w.sum() * (n - 1)).astype(np.int64)
    founder = first[np.searchsorted(first, np.arange(n), side="right") - 1]
    s = np.arange(1, n)
    f = founder[1:]
    parent[1:] = np.where(s == f, 0, f + (rng.random(n - 1) * (s - f)).astype(np.int64))
    return parent


def _values(n, nq, kmers, s64, tree, seed):
    """Bin values int16 [n + nq, K, 64 * s64] on the device: a population of n
    samples and nq queries, each query a descendant of a random sample."""
    rng = np.random.default_rng(seed)
    parent = _tree(n, tree == "clades", rng)
    if nq:
        parent = np.concatenate([parent, rng.integers(0, n, nq)])
    m = n + nq
    k = np.asarray(kmers, np.float64)[None, :]
    c, a = rng.uniform(0, 0.03, m)[:, None], rng.uniform(0, 0.2, m)[:, None]
    p = torch.from_numpy((1.0 - (1.0 - c) ** k * (1.0 - a)).astype(np.float32)).to(DEVICE)
    level = np.zeros(m, np.int64)
    for s in range(m):
        if parent[s] >= 0:
            level[s] = level[parent[s]] + 1
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    out = torch.empty((m, len(kmers), 64 * s64), dtype=torch.int16, device=DEVICE)
    step = max(1, (1 << 27) // (len(kmers) * 64 * s64))
    for lv in range(int(level.max()) + 1):
        idx = np.flatnonzero(level == lv)
        for i in range(0, len(idx), step):
            part = idx[i:i + step]
            at = torch.from_numpy(part).to(DEVICE)
            shape = (len(part),) + tuple(out.shape[1:])
            fresh = torch.randint(0, 1 << BBITS, shape, dtype=torch.int16, device=DEVICE,
                                  generator=gen)
            if lv > 0:
                u = torch.rand(shape, dtype=torch.float32, device=DEVICE, generator=gen)
                old = out[torch.from_numpy(parent[part]).to(DEVICE)]
                fresh = torch.where(u < p[at][:, :, None], fresh, old)
            out[at] = fresh
    return out


def _words(vals):
    """Bin values -> the library's sketch words int64 [m, K, s64 * 14]: bit i of
    word (block * 14 + plane) is bit `plane` of bin 64 * block + i."""
    m, K, bins = vals.shape
    out = torch.empty((m, K, bins // 64, BBITS), dtype=torch.int64, device=vals.device)
    place = torch.ones(64, dtype=torch.int64, device=vals.device) << torch.arange(
        64, device=vals.device)
    step = max(1, (1 << 26) // (K * bins))
    for i in range(0, m, step):
        v = vals[i:i + step].view(-1, K, bins // 64, 64)
        for b in range(BBITS):
            out[i:i + step, :, :, b] = (((v >> b) & 1).to(torch.int64) * place).sum(-1)
    return out.view(m, K, bins // 64 * BBITS)


def _info(m, seed):
    """Genome lengths and random-match clusters of m samples."""
    rng = np.random.default_rng(seed + 77)
    return rng.integers(1_800_000, 3_200_000, m).astype(np.uint64), rng.integers(0, 3, m).astype(
        np.uint16)


def _table(kmers, seed):
    """A 3-cluster Monte Carlo table: chances falling with k."""
    rng = np.random.default_rng(seed + 78)
    t = 0.1 * rng.random((len(kmers), 3, 3)) * np.exp(-0.35 * (np.asarray(kmers) - 13))[:, None, None]
    return t.astype(np.float32)


def _model(ctx, case, kmers, seed):
    if case["random"] == "table":
        return capi.Random(ctx, capi.RANDOM_TABLE, kmers, True, _table(kmers, seed))
    if case["random"] == "equal":
        return capi.Random(ctx, capi.RANDOM_EQUAL_BASE, kmers, True)
    return None


def _database(ctx, words, kmers, s64, lens, clusters):
    torch.cuda.synchronize()      # the library reads the words on its own stream
    return capi.Database(ctx, words.data_ptr(), kmers, s64, n_samples=words.shape[0],
                         cluster=clusters, seq_len=lens)


def _pinned(t):
    """A page-locked host copy of a device tensor as uint64 numpy."""
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h, h.numpy().view(np.uint64)


OUT = {"core_acc": capi.OUT_CORE_ACC, "jaccard": capi.OUT_JACCARD, "counts": capi.OUT_COUNTS}


def _out_tensor(pairs, K, out):
    if out == "core_acc":
        return torch.empty((pairs, 2), dtype=torch.float32, device=DEVICE)
    return torch.empty((pairs, K), dtype=torch.float32 if out == "jaccard" else torch.int32,
                       device=DEVICE)


def _batch_jobs(case, seed):
    """Databases of 50 .. 2,500 samples, k sets of 4 .. 14 odd lengths, four
    sketch widths; half all-vs-all, half a tenth of the samples as queries."""
    rng = np.random.default_rng(40_000 + case["n"])     # the shapes belong to the case
    jobs = []
    for j in range(case["n"]):
        n = int(round(math.exp(rng.uniform(math.log(50), math.log(2500)))))
        K = int(rng.integers(4, 15))
        kmers = sorted(int(k) for k in rng.choice(np.arange(13, 40, 2), K, replace=False))
        s64 = int(rng.choice([16, 64, 156, 312]))
        jobs.append(dict(n=n, nq=0 if rng.random() < 0.5 else max(1, n // 10), kmers=kmers,
                         s64=s64, seed=seed * 64 + j))
    return jobs


def _genome(length, gen):
    """Bases (ASCII) at GC 0.38."""
    u = torch.rand(length, device=DEVICE, generator=gen)
    code = torch.bucketize(u, torch.tensor([0.31, 0.50, 0.69], device=DEVICE))
    return torch.tensor([65, 67, 71, 84], dtype=torch.uint8, device=DEVICE)[code]


def _genomes(n, length, seed):
    """Related genomes: each copies an earlier one with up to 0.4% changed bases
    and up to 3% of it replaced."""
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    rng = np.random.default_rng(seed)
    out = torch.empty((n, length), dtype=torch.uint8, device=DEVICE)
    out[0] = _genome(length, gen)
    for g in range(1, n):
        out[g] = out[int(rng.integers(0, g))]
        fresh = _genome(length, gen)
        snp = torch.rand(length, device=DEVICE, generator=gen) < rng.uniform(0, 0.004)
        out[g] = torch.where(snp, fresh, out[g])
        seg = min(5000, length // 8)
        for _ in range(int(rng.uniform(0, 0.03) * length / seg)):
            s = int(rng.integers(0, length - seg))
            out[g, s:s + seg] = fresh[s:s + seg]
    return out


def _read_set(length, seed):
    """150-base reads at 10x coverage of one genome with 1% errors."""
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    genome = _genome(length, gen)
    n_reads = 10 * length // 150
    start = torch.randint(0, length - 150, (n_reads, 1), device=DEVICE, generator=gen)
    reads = genome[start + torch.arange(150, device=DEVICE)]
    wrong = torch.rand(reads.shape, device=DEVICE, generator=gen) < 0.01
    return torch.where(wrong, _genome(reads.numel(), gen).view(reads.shape), reads)


# ------------------------------------------------------------ prepare / run

def prepare(case, seed):
    ctx, kind = _ctx(), case["kind"]
    kmers = _kmers(case)
    st = dict(kind=kind, ctx=ctx, case=case)
    if kind == "batch":
        jobs, st["keep"], st["outs"] = [], [], []
        for j in _batch_jobs(case, seed):
            w = _words(_values(j["n"], j["nq"], j["kmers"], j["s64"], "random", j["seed"]))
            ref = _database(ctx, w[:j["n"]], j["kmers"], j["s64"], None, None)
            qry = _database(ctx, w[j["n"]:], j["kmers"], j["s64"], None, None) if j["nq"] else None
            pairs = j["nq"] * j["n"] if j["nq"] else j["n"] * (j["n"] - 1) // 2
            st["outs"].append(_out_tensor(pairs, len(j["kmers"]), "core_acc"))
            jobs.append((ref, qry, None, capi.OUT_CORE_ACC, st["outs"][-1].data_ptr()))
        torch.cuda.synchronize()
        st["batch"] = capi.Batch(ctx, jobs)
        return st
    if kind == "sketch":
        n, L = case["n"], case["length"]
        st["bases"] = _genomes(n, L, seed)
        st["off"] = np.arange(n + 1, dtype=np.int64) * L
        st["ss"] = np.arange(n + 1, dtype=np.int64)
        st["words"] = torch.empty((n, len(kmers), case["s64"] * BBITS), dtype=torch.int64,
                                  device=DEVICE)
        st["inv"] = torch.empty((n, len(kmers)), dtype=torch.float64, device=DEVICE)
        st["dens"] = torch.empty(n, dtype=torch.uint8, device=DEVICE)
        torch.cuda.synchronize()
        return st
    if kind == "reads":
        sets = [_read_set(case["length"], seed * 16 + i) for i in range(case["n"])]
        st["hold"] = torch.empty(sum(r.numel() for r in sets), dtype=torch.uint8, pin_memory=True)
        st["hold"].copy_(torch.cat([r.view(-1) for r in sets]))
        st["bases"] = st["hold"].numpy()
        per = sets[0].shape[0]
        st["off"] = np.arange(case["n"] * per + 1, dtype=np.int64) * 150
        st["ss"] = np.arange(case["n"] + 1, dtype=np.int64) * per
        return st
    n, nq, s64 = case["n"], case["nq"], case["s64"]
    words = _words(_values(n, nq, kmers, s64, case["tree"], seed))
    lens, cl = _info(n + nq, seed)
    st["rnd"] = _model(ctx, case, kmers, seed)
    if kind == "host":
        st["hold"], w = _pinned(words)
        pairs = nq * n if nq else n * (n - 1) // 2
        st["out_t"] = torch.empty((pairs, 2), dtype=torch.float32, pin_memory=True)
        st["args"] = dict(ref_words=w[:n], query_words=w[n:] if nq else None, kmers=kmers,
                          sketchsize64=s64, ref_cluster=cl[:n], ref_seq_len=lens[:n],
                          query_cluster=cl[n:] if nq else None,
                          query_seq_len=lens[n:] if nq else None, random=st["rnd"],
                          out=st["out_t"].numpy())
        return st
    st["ref"] = _database(ctx, words[:n], kmers, s64, lens[:n], cl[:n])
    if kind == "self":
        st["out"] = _out_tensor(n * (n - 1) // 2, len(kmers), case["out"])
    elif kind in ("query", "query_knn"):
        st["query"] = _database(ctx, words[n:], kmers, s64, lens[n:], cl[n:])
        if kind == "query":
            st["out"] = _out_tensor(nq * n, len(kmers), case["out"])
    elif kind == "serve":
        st["hold"], st["qwords"] = _pinned(words[n:])
        st["info"] = (cl[n:], lens[n:])
        st["server"] = capi.Server(ctx, st["ref"], st["rnd"], slots=2, slice_queries=256,
                                   kNN=case["knn"])
    torch.cuda.synchronize()
    return st


def run(st):
    ctx, kind, case = st["ctx"], st["kind"], st["case"]
    if kind in ("self", "query"):
        capi.dists_dense(ctx, st["ref"], st.get("query"), st["rnd"], OUT[case["out"]],
                         st["out"].data_ptr())
        return st["out"]
    if kind == "query_knn":
        return capi.query_knn(ctx, st["ref"], st["query"], case["knn"], random=st["rnd"])
    if kind == "knn":
        _, j, d = capi.dists_knn(ctx, st["ref"], case["knn"], random=st["rnd"])
        return j, d
    if kind == "serve":
        t = st["server"].submit(st["qwords"], *st["info"])
        st["server"].wait(t)
        return st["server"].result(t)[:2]
    if kind == "host":
        return capi.query_db(ctx, **st["args"])
    if kind == "batch":
        st["batch"].run()
        return st["outs"]
    if kind == "sketch":
        capi.sketch_device(ctx, st["bases"].data_ptr(), st["off"], st["ss"], _kmers(case),
                           case["s64"], st["words"].data_ptr(),
                           d_inv_minhash=st["inv"].data_ptr(), d_densified=st["dens"].data_ptr())
        return st["words"], st["inv"], st["dens"]
    words, inv, dens = capi.sketch(ctx, st["bases"], st["off"], st["ss"], _kmers(case),
                                   case["s64"], min_count=3)
    return words.view(np.int64), inv, dens


# ------------------------------------------------------------------- exact

def _exact_dists(vals, n, nq, kmers, case, seed, out):
    """[pairs, 2] core/accessory or [pairs, K] Jaccards in float64: the bins in
    common, the random-match correction, and the log-linear fit over the
    k-mer lengths from the first to the last Jaccard above tolerance."""
    K, bins = len(kmers), vals.shape[2]
    ref, rows = vals[:n], vals[n:] if nq else vals[:n]
    cnt = []
    for i in range(rows.shape[0]):
        col0 = 0 if nq else i + 1
        cnt.append((ref[col0:] == rows[i]).sum(-1, dtype=torch.int32))
    cnt = torch.cat(cnt).to(torch.float64)
    obs = cnt / bins
    lens, cl = _info(n + nq, seed)
    if nq:
        qi = torch.arange(nq, device=DEVICE).repeat_interleave(n) + n
        ri = torch.arange(n, device=DEVICE).repeat(nq)
    else:
        i, j = np.triu_indices(n, 1)
        ri, qi = torch.from_numpy(i).to(DEVICE), torch.from_numpy(j).to(DEVICE)
    r = torch.zeros_like(obs)
    if case["random"] == "table":
        t = torch.from_numpy(_table(kmers, seed)).to(DEVICE).to(torch.float64)
        c = torch.from_numpy(cl.astype(np.int64)).to(DEVICE)
        for k in range(K):
            r[:, k] = t[k][c[ri], c[qi]]
    elif case["random"] == "equal":
        ln = torch.from_numpy(lens.astype(np.float64)).to(DEVICE)
        for k in range(K):
            miss = math.log1p(-0.5 ** (2 * (kmers[k] - 1) + 1))
            p = -torch.expm1(ln * miss)
            r[:, k] = p[ri] * p[qi] / (p[ri] + p[qi] - p[ri] * p[qi])
    jac = (obs - r).clamp(min=0) / (1 - r)
    if out == "counts":
        return cnt
    if out == "jaccard":
        return jac
    jac = jac.to(torch.float32).to(torch.float64)     # the fit takes single-precision Jaccards
    ok = jac > 5.0 / bins
    pos = torch.arange(K, device=DEVICE)
    first = torch.where(ok, pos, K).amin(1, keepdim=True)
    last = torch.where(ok, pos, -1).amax(1, keepdim=True)
    used = (pos >= first) & (pos <= last)
    w = used.to(torch.float64)
    num = w.sum(1)
    x = torch.tensor(kmers, dtype=torch.float64, device=DEVICE)
    bad = (num < 2) | (used & (jac <= 0)).any(1)
    y = torch.where(used & (jac > 0), jac, torch.ones_like(jac)).log()
    num = num.clamp(min=1)
    xm, ym = (w * x).sum(1) / num, (w * y).sum(1) / num
    dx = w * (x - xm[:, None])
    slope = (dx * y).sum(1) / (dx * dx).sum(1).clamp(min=1e-300)
    icpt = ym - slope * xm
    res = torch.stack([-torch.expm1(slope.clamp(max=0)), -torch.expm1(icpt.clamp(max=0))], 1)
    res[bad] = 0
    return res


def exact(case, seed):
    kind = case["kind"]
    if kind in ("sketch", "reads"):
        return None
    if kind == "batch":
        jobs = _batch_jobs(case, seed)
        if sum(_comparisons(j["n"], j["nq"], len(j["kmers"]), j["s64"]) for j in jobs) > EXACT_LIMIT:
            return None
        return [_exact_dists(_values(j["n"], j["nq"], j["kmers"], j["s64"], "random", j["seed"]),
                             j["n"], j["nq"], j["kmers"], dict(random="none"), j["seed"],
                             "core_acc") for j in jobs]
    n, nq, kmers = case["n"], case["nq"], _kmers(case)
    if _comparisons(n, nq, case["K"], case["s64"]) > EXACT_LIMIT or case["out"] == "counts":
        return None
    vals = _values(n, nq, kmers, case["s64"], case["tree"], seed)
    d = _exact_dists(vals, n, nq, kmers, case, seed, case["out"])
    if kind in ("self", "query", "host"):
        return d
    if kind == "knn":
        i, j = np.triu_indices(n, 1)
        sq = torch.full((n, n), math.inf, dtype=torch.float64, device=DEVICE)
        ii, jj = torch.from_numpy(i).to(DEVICE), torch.from_numpy(j).to(DEVICE)
        sq[ii, jj] = d[:, 0]
        sq[jj, ii] = d[:, 0]
        return None, sq.sort(1).values[:, :case["knn"]].reshape(-1)
    return None, d[:, 0].view(nq, n).sort(1).values[:, :case["knn"]]


# -------------------------------------------------------------------- work

def _comparisons(n, nq, K, s64):
    return (nq * n if nq else n * (n - 1) // 2) * K * 64.0 * s64


def _dist_work(n, nq, K, s64, out_bytes):
    """Each sketch read once, each result written once; an operation is one
    comparison of two bins."""
    return {"bytes": (n + nq) * K * s64 * BBITS * 8.0 + out_bytes,
            "flops": _comparisons(n, nq, K, s64)}


def work(case):
    kind, n, nq, K, s64 = (case[x] for x in ("kind", "n", "nq", "K", "s64"))
    if kind == "batch":
        w = {"bytes": 0.0, "flops": 0.0}
        for j in _batch_jobs(case, 0):
            pairs = j["nq"] * j["n"] if j["nq"] else j["n"] * (j["n"] - 1) // 2
            one = _dist_work(j["n"], j["nq"], len(j["kmers"]), j["s64"], 8.0 * pairs)
            w = {x: w[x] + one[x] for x in w}
        return w
    if kind in ("sketch", "reads"):
        # each base read once, each sketch written once; an operation is one
        # window hashed
        bases = n * case["length"] * (1 if kind == "sketch" else 10)
        return {"bytes": bases + n * K * (s64 * BBITS * 8.0 + 8), "flops": float(bases * K)}
    pairs = nq * n if nq else n * (n - 1) // 2
    if kind in ("knn", "query_knn", "serve"):
        return _dist_work(n, nq, K, s64, (nq or n) * case["knn"] * 12.0)
    per = 8.0 if case["out"] == "core_acc" else 4.0 * K
    return _dist_work(n, nq, K, s64, pairs * per)
