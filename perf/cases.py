"""The calls this engine's performance is judged by: searches, serving and exact scans over loaded
indices, from one query on a small index to 10,000 queries on a million rows.

A user of the engine keeps one loaded index and sends it new queries, so the database and its
graph belong to the case and the queries come from the seed. The index files are written here: the
engine's own multi-threaded builders (and the reference's) link a graph in an order that depends on
timing, and two processes that compare results need the same graph. Construction itself is left
out for the same reason: two builds of one database give different graphs.

A graph has the reference's shape: geometric levels, up to M neighbours per node chosen from the
nearest candidates by the keep-if-closer rule, links made both ways, at most M (upper levels) and
2M (level 0) per node.
"""
import ctypes
import functools
import math
import os
import tempfile

import numpy as np
import torch

import nmslib_b200 as nmslib
from nmslib_b200 import _capi
from nmslib_b200.serving import Server

SIFT = "l2sqr_sift"
SPACES = ("l2", "cosinesimil", "negdotprod", "l1", "linf", SIFT)
SERVE_MAX = 256      # largest request of the serving mix
SERVE_REQUESTS = 24  # requests in flight at once


def listed():
    return [
        # an interactive lookup: one query on a small index that sits in L2 (latency and launches)
        dict(name="one_query_10k", call="one", space="l2", n=10_000, dim=128, m=16, nq=1, k=10, ef=100),
        # a request of a handful of queries against the million-row index (latency of one search)
        dict(name="request16_1m", call="batch", space="l2", n=1_000_000, dim=128, m=16, nq=16, k=10, ef=100),
        # an application's batch over a small index: the 10K x 128 configuration with its 1,000 queries
        dict(name="batch1k_10k", call="batch", space="l2", n=10_000, dim=128, m=16, nq=1_000, k=10, ef=100),
        # the benchmark's batch: 10,000 queries over 1M x 128 rows at efSearch 64
        dict(name="batch10k_1m", call="batch", space="l2", n=1_000_000, dim=128, m=16, nq=10_000, k=10, ef=64),
        # an offline pipeline with queries and results on the GPU, high recall, long result lists
        dict(name="device10k_1m_ef256", call="device", space="l2", n=1_000_000, dim=128, m=16, nq=10_000, k=100,
             ef=256),
        # word-embedding search: 100-float rows (not a multiple of 16), M 24, high recall
        dict(name="cosine10k_1m_d100", call="batch", space="cosinesimil", n=1_000_000, dim=100, m=24, nq=10_000, k=10,
             ef=200),
        # a service's collected calls with their own k and efSearch, wide rows, both algorithms
        dict(name="mixed2k_200k_d960", call="mixed", space="negdotprod", n=200_000, dim=960, m=16, nq=2_000, k=100,
             ef=1024),
        # L1 search over feature vectors with an odd row length and an odd batch
        dict(name="l1_3001_200k_d100", call="batch", space="l1", n=200_000, dim=100, m=16, nq=3_001, k=10, ef=100),
        # byte descriptors with integer distances
        dict(name="sift_u8_5k_500k", call="batch", space=SIFT, n=500_000, dim=128, m=16, nq=5_000, k=10, ef=100),
        # the continuous-batching server: requests of 1 to 256 queries with two k and two efSearch
        dict(name="serve24_1m", call="serve", space="l2", n=1_000_000, dim=128, m=16, nq=SERVE_MAX, k=100, ef=400),
        # exact neighbours of a whole query set (ground truth, re-ranking without a graph)
        dict(name="exact10k_1m", call="exact", space="l2", n=1_000_000, dim=128, m=16, nq=10_000, k=10, ef=0),
        # exact neighbours of a few queries, odd sizes
        dict(name="exact333_1m_d100", call="exact", space="cosinesimil", n=1_000_000, dim=100, m=24, nq=333, k=32,
             ef=0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["one", "batch", "batch", "batch", "batch", "device", "mixed", "serve", "exact"])
    space = rng.choice({"batch": SPACES, "one": SPACES, "exact": SPACES[:3], "serve": SPACES[:3],
                        "device": SPACES[:3], "mixed": SPACES[:3]}[call])
    wide = rng.random() < 0.2 and space in SPACES[:3]
    dim = 128 if space == SIFT else _log_int(rng, 257, 1024) if wide else _log_int(rng, 16, 256)
    if space != SIFT and rng.random() < 0.5:
        dim = max(16, dim // 16 * 16)  # the row lengths of real data sets are often multiples of 16
    n = _log_int(rng, 5_000, 200_000 if wide else 1_000_000)
    nq = 1 if call == "one" else SERVE_MAX if call == "serve" else _log_int(rng, 2, 2_000 if wide else 10_000)
    k = rng.randint(1, 32) if call == "exact" else _log_int(rng, 1, 100)
    ef = 0 if call == "exact" else _log_int(rng, 16, 400)
    if call == "mixed":
        k, ef = 100, 1024
    return dict(call=call, space=space, n=n, dim=dim, m=rng.choice([8, 16, 24, 32]), nq=nq, k=k, ef=ef)


# ------------------------------------------------------------------ data
def _generator(*key):
    """A generator on the GPU whose stream is a function of the key alone."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(np.random.SeedSequence([int.from_bytes(str(x).encode(), "little") % (1 << 62) for x in key])
                      .generate_state(1, np.uint64)[0] >> 1))
    return g


def _centres(space, n, dim):
    g = _generator("centres", space, n, dim)
    c = torch.randn((max(16, n // 1000), dim), generator=g, device="cuda")
    if space in ("l2", SIFT):
        c = (c * 40).abs().clamp(max=255).round()
    elif space == "cosinesimil":
        c *= torch.rand(dim, generator=g, device="cuda") * 1.5 + 0.5
    elif space == "negdotprod":
        c = c.abs()
    return c


def _points(space, c, rows, g):
    """`rows` vectors around the centres, and the centre of each: integer-valued SIFT-like rows for
    l2 (so equal distances happen), scaled Gaussians for cosine, absolute ones for the dot product."""
    z = torch.randint(0, c.shape[0], (rows,), generator=g, device="cuda")
    e = torch.randn((rows, c.shape[1]), generator=g, device="cuda")
    if space in ("l2", SIFT):
        x = (c[z] + 12 * e).round().clamp(0, 255)
    elif space == "negdotprod":
        x = (c[z] + 0.5 * e).abs()
    else:
        x = c[z] + 0.5 * e
    return x, z


def _base(space, n, dim):
    x, z = _points(space, _centres(space, n, dim), n, _generator("base", space, n, dim))
    return (torch.nn.functional.normalize(x) if space == "cosinesimil" else x), z


def _queries(case, seed, rows):
    c = _centres(case["space"], case["n"], case["dim"])
    q = _points(case["space"], c, rows, _generator("queries", seed))[0]
    return q.to(torch.uint8) if case["space"] == SIFT else q


# ------------------------------------------------------------------ graph
def _dist(space, a, b):
    """Distances [..., p, q] between rows a [..., p, d] and b [..., q, d]. L1 and LInf graphs are
    built by squared L2, which orders neighbours closely enough to search by either."""
    dot = a @ b.transpose(-1, -2)
    if space == "negdotprod":
        return -dot
    return (a * a).sum(-1)[..., :, None] + (b * b).sum(-1)[..., None, :] - 2 * dot


def _order_key(d, ids):
    """int64 keys ordered by (distance, id): unique, so a selection has one answer."""
    i = d.view(torch.int32)
    return ((i ^ ((i >> 31) & 0x7FFFFFFF)).to(torch.int64) << 32) | ids


def _nearest(space, x, rows, cand, kk):
    """The kk nearest of `cand` for each of `rows` (ids), nearest first: (ids, distances)."""
    d = _dist(space, x[rows], x[cand])
    key = _order_key(d, cand)
    key[rows[:, None] == cand] = torch.iinfo(torch.int64).max
    key = key.topk(kk, largest=False).values
    i = (key >> 32).to(torch.int32)
    return key & 0x7FFFFFFF, (i ^ ((i >> 31) & 0x7FFFFFFF)).view(torch.float32)


def _candidates(space, x, z, rows, pool, kk):
    """The kk nearest of `pool` for each of `rows`: among all of them, or for a large pool among the
    clusters around each row's own."""
    ids = torch.empty((len(x), kk), dtype=torch.int64, device="cuda")
    d = torch.empty((len(x), kk), device="cuda")
    if len(pool) <= 16_384:
        parts = [(r, pool) for r in rows.split(4096)]
    else:
        def by_cluster(nodes):
            order = nodes[torch.argsort(z[nodes], stable=True)]
            return order.split(torch.bincount(z[nodes], minlength=int(z.max()) + 1).tolist())
        members, asking = by_cluster(pool), by_cluster(rows)
        full = [c for c, r in enumerate(members) if len(r)]
        mean = torch.stack([x[members[c]].mean(0) for c in full])
        near = torch.cdist(mean, mean).topk(min(len(full), 3 + 1500 * len(full) // len(pool)), largest=False).indices
        parts = [(asking[c], torch.cat([members[c]] + [members[full[o]] for o in near[i].tolist() if full[o] != c]))
                 for i, c in enumerate(full) if len(asking[c])]
    for r, cand in parts:
        ids[r], d[r] = _nearest(space, x, r, cand, kk)
    return ids[rows], d[rows]


def _select(space, x, cand, d, m):
    """The reference's second heuristic over sorted candidates: keep one unless a kept one is closer
    to it than the node itself, up to m. A mask of `cand`."""
    keep = torch.zeros(cand.shape, dtype=torch.bool, device="cuda")
    step = max(1024, (1 << 28) // (cand.shape[1] * x.shape[1]))
    for lo in range(0, len(cand), step):
        v = x[cand[lo:lo + step]]
        g = _dist(space, v, v)
        kept, dn = keep[lo:lo + step], d[lo:lo + step]
        for i in range(cand.shape[1]):
            closer = (kept & (g[:, i] < dn[:, i:i + 1])).any(1)
            kept[:, i] = ~closer & (kept.sum(1) < m)
    return keep


def _links(space, x, z, nodes, m, cap):
    """Neighbour lists of one level: ids [len(nodes), cap] padded with -1, and their lengths. Nodes
    choose among those inserted before them, as in the reference: the first few hundred among
    themselves, then each doubling among all that came before it and itself, so that early nodes
    carry the long links. A list past `cap` is cut by the same heuristic."""
    n = len(nodes)
    out = torch.full((n, cap), -1, dtype=torch.int32, device="cuda")
    if n < 2:
        return out, torch.zeros(n, dtype=torch.int32, device="cuda")
    row = torch.zeros(len(x), dtype=torch.int64, device="cuda")
    row[nodes] = torch.arange(n, device="cuda")
    edges, lo, hi = [], 0, min(n, 256)
    while lo < n:
        cand, d = _candidates(space, x, z, nodes[lo:hi], nodes[:hi], min(6 * m, 128, n - 1))
        keep = _select(space, x, cand, d, m)
        u = torch.arange(lo, hi, device="cuda")[:, None].expand_as(cand)[keep]
        edges.append((u, row[cand[keep]], d[keep]))
        lo, hi = hi, min(n, 2 * hi)
    u, v, d = (torch.cat(e) for e in zip(*edges))
    back = ~torch.isin(v * n + u, u * n + v)
    late = torch.cat([torch.zeros_like(u), torch.ones_like(u[back])])
    src, dst, d = torch.cat([u, v[back]]), torch.cat([v, u[back]]), torch.cat([d, d[back]])

    def by(*keys):  # sorts the edges by the last key, ties by the one before it, and so on
        o = torch.arange(len(src), device="cuda")
        for key in keys:
            o = o[torch.argsort(key[o], stable=True)]
        count = torch.bincount(src, minlength=n)
        return src[o], dst[o], d[o], torch.arange(len(src), device="cuda") - (count.cumsum(0) - count)[src[o]], count

    # own links and the nearest links back, up to 96, then in order of distance
    src, dst, d, place, _ = by(_order_key(d, dst), 2 * src + late)
    src, dst, d = src[place < 96], dst[place < 96], d[place < 96]
    src, dst, d, place, count = by(_order_key(d, dst), src)
    over = torch.nonzero(count > cap).flatten()
    if len(over):
        slot = torch.full((n,), -1, dtype=torch.int64, device="cuda")
        slot[over] = torch.arange(len(over), device="cuda")
        e = torch.nonzero(slot[src] >= 0).flatten()
        cand = nodes[src.new_zeros(len(over), 96)]
        cd = torch.full((len(over), 96), math.inf, device="cuda")
        cand[slot[src[e]], place[e]], cd[slot[src[e]], place[e]] = nodes[dst[e]], d[e]
        keep = _select(space, x, cand, cd, cap) & (cd < math.inf)
        stay = slot[src] < 0
        stay[e] = keep[slot[src[e]], place[e]]
        src, dst, d = src[stay], dst[stay], d[stay]
        src, dst, d, place, count = by(_order_key(d, dst), src)
    out[src, place] = nodes[dst].to(torch.int32)
    return out, count.to(torch.int32)


def _graph(space, n, dim, m):
    """(rows, per-node level, entry point, [(nodes, lists, lengths) of each level])."""
    x, z = _base(space, n, dim)
    u = torch.rand(n, generator=_generator("levels", n, m), device="cuda", dtype=torch.float64)
    level = (-(1 - u).log() / math.log(m)).long()
    levels = []
    for lev in range(int(level.max()) + 1):
        nodes = torch.nonzero(level >= lev).flatten()
        levels.append((nodes, *_links(space, x, z, nodes, m, 2 * m if lev == 0 else m)))
    return x, level, int(torch.argmax(level)), levels


# ------------------------------------------------------------------ index files
def _write_optimized(path, space, x, level, entry, levels, m):
    """The reference's optimized layout: header, one packed row per node, then the upper lists."""
    n, dim = x.shape
    _, lists, count = levels[0]
    row = torch.zeros((n, 4 + dim + 1 + 2 * m), dtype=torch.int32, device="cuda")
    row[:, 0] = torch.arange(n, device="cuda")
    row[:, 1] = -1
    row[:, 2] = 4 * dim
    row[:, 4:4 + dim] = x.view(torch.int32)
    row[:, 4 + dim] = count
    row[:, 5 + dim:] = lists.clamp(min=0)
    size = level * (m + 1)
    start = (size + 1).cumsum(0) - (size + 1)
    upper = torch.zeros(int((size + 1).sum()), dtype=torch.int32, device="cuda")
    upper[start] = 4 * size.to(torch.int32)
    for lev, (nodes, lists, count) in enumerate(levels[1:]):
        at = start[nodes] + 1 + lev * (m + 1)
        upper[at] = count
        upper[at[:, None] + 1 + torch.arange(m, device="cuda")] = lists.clamp(min=0)
    code = {"l2": 1 if dim % 16 == 0 else 2, "cosinesimil": 3, "negdotprod": 4, "l1": 5, "linf": 6}[space]
    with open(path, "wb") as f:
        f.write(np.array([1, n], np.uint32).tobytes())
        f.write(np.array([4 * row.shape[1], 16 + 4 * dim, 0], np.uint64).tobytes())
        f.write(np.array([len(levels) - 1, entry], np.int32).tobytes())
        f.write(np.array([m, 2 * m], np.uint64).tobytes())
        f.write(np.int32(code).tobytes() + np.uint64(3).tobytes())
        for part in row.split(1 << 17):
            f.write(part.cpu().numpy().tobytes())
        f.write(upper.cpu().numpy().tobytes())


def _write_sift(path, x, level, entry, levels, m):
    """The regular graph file and the objects file, the form l2sqr_sift indices are saved in."""
    n = len(x)
    count = torch.zeros((n, len(levels)), dtype=torch.int64, device="cuda")
    for lev, (nodes, _, c) in enumerate(levels):
        count[nodes, lev] = 1 + c.to(torch.int64)
    size = 1 + count.sum(1)
    start = size.cumsum(0) - size
    words = torch.zeros(int(size.sum()), dtype=torch.int32, device="cuda")
    words[start] = level.to(torch.int32)
    for lev, (nodes, lists, c) in enumerate(levels):
        at = (start + 1 + count[:, :lev].sum(1))[nodes]
        words[at] = c
        u, j = torch.nonzero(lists >= 0, as_tuple=True)
        words[at[u] + 1 + j] = lists[u, j]
    with open(path, "wb") as f:
        f.write(np.array([0, n, len(levels) - 1, entry], np.uint32).tobytes())
        f.write(np.array([m, m, 2 * m], np.uint64).tobytes())
        f.write(words.cpu().numpy().tobytes())
    rec = np.zeros(n, dtype=[("len", "<u8"), ("id", "<i4"), ("label", "<i4"), ("dlen", "<u8"), ("v", "u1", 128),
                             ("norm", "<i4")])
    rec["len"], rec["id"], rec["label"], rec["dlen"] = 148, np.arange(n), -1, 132
    rec["v"], rec["norm"] = x.to(torch.uint8).cpu().numpy(), (x * x).sum(1).to(torch.int32).cpu().numpy()
    with open(path + ".dat", "wb") as f:
        f.write(np.uint64(n).tobytes() + rec.tobytes())


@functools.lru_cache(maxsize=8)
def _index(space, n, dim, m):
    """A loaded index, kept as a program keeps it from one batch of queries to the next."""
    graph = _graph(space, n, dim, m)
    with tempfile.TemporaryDirectory(dir="/dev/shm" if os.path.isdir("/dev/shm") else None) as tmp:
        path = os.path.join(tmp, "index")
        if space == SIFT:
            index = nmslib.init(method="hnsw", space=SIFT, data_type=nmslib.DataType.DENSE_UINT8_VECTOR,
                                dtype=nmslib.DistType.INT)
            _write_sift(path, *graph, m)
            index.loadIndex(path, load_data=True)
        else:
            index = nmslib.init(method="hnsw", space=space)
            _write_optimized(path, space, *graph, m)
            index.loadIndex(path)
    return index


@functools.lru_cache(maxsize=2)
def _server(space, n, dim, m):
    return Server(_index(space, n, dim, m), memory_budget_bytes=8 << 30, max_batch=SERVE_MAX, max_k=100)


# ------------------------------------------------------------------ cases
def _requests(case):
    """The serving mix: sizes log-uniform in 1..256, k and efSearch low or high."""
    rng = np.random.default_rng([case[name] for name in ("n", "dim", "m", "k", "ef")])
    sizes = np.minimum(case["nq"], np.floor(np.exp(rng.uniform(0, np.log(case["nq"] + 1), SERVE_REQUESTS)))).astype(int)
    sizes[0] = case["nq"]
    ks = rng.choice([min(10, case["k"]), case["k"]], SERVE_REQUESTS)
    efs = rng.choice([max(1, case["ef"] // 4), case["ef"]], SERVE_REQUESTS)
    return sizes.tolist(), ks.tolist(), efs.tolist()


def prepare(case, seed):
    key = case["space"], case["n"], case["dim"], case["m"]
    index = _index(*key)
    state = dict(call=case["call"], index=index, k=case["k"], ef=case["ef"])
    if case["call"] == "serve":
        sizes, ks, efs = _requests(case)
        q = _queries(case, seed, sum(sizes)).cpu().numpy()
        state.update(server=_server(*key), ks=ks, efs=efs, q=np.split(q, np.cumsum(sizes)[:-1]))
        return state
    q = _queries(case, seed, case["nq"])
    if case["call"] == "device":
        nq, k = case["nq"], case["k"]
        state.update(q=q.contiguous(), ids=torch.empty((nq, k), dtype=torch.int32, device="cuda"),
                     dists=torch.empty((nq, k), device="cuda"), counts=torch.empty(nq, dtype=torch.int32, device="cuda"))
        return state
    state["q"] = q.cpu().numpy()
    if case["call"] == "mixed":
        rng = np.random.default_rng([11, seed])
        state["k"] = rng.choice([1, 10, 100], case["nq"]).astype(np.int32)
        state["ef"] = rng.integers(64, case["ef"] + 1, case["nq"]).astype(np.int32)
    return state


def run(state):
    call, index, q, k = state["call"], state["index"], state["q"], state["k"]
    if call == "exact":
        return index.bruteForceBatchArrays(q, k)
    if call == "mixed":
        return index.knnQueryBatchArrays(q, k, ef=state["ef"])
    if call == "serve":
        server = state["server"]
        sent = [server.submit(*request) for request in zip(q, state["ks"], state["efs"])]
        return [server.wait(r)[:2] for r in sent]
    index.setQueryTimeParams({"efSearch": state["ef"]})
    if call == "one":
        return index.knnQuery(q[0], k)
    if call == "device":  # the C ABI on device buffers, on the caller's stream
        ptr = [ctypes.c_void_p(state[name].data_ptr()) for name in ("q", "ids", "dists", "counts")]
        _capi.check(_capi.load().nmsg_knn_batch(
            index._require(), ptr[0], q.shape[0], q.shape[1], k, None, None, k, *ptr[1:], None,
            _capi.FLAG_DEVICE_PTRS, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return state["ids"], state["dists"], state["counts"]
    return index.knnQueryBatchArrays(q, k)


def exact(case, seed):
    """The exact scans in 64 bits. A graph search's distances have no value apart from the walk that
    found them, so those calls have none."""
    if case["call"] != "exact":
        return None
    x = _base(case["space"], case["n"], case["dim"])[0].double()
    q = _queries(case, seed, case["nq"]).double()
    if case["space"] == "cosinesimil":
        q = torch.nn.functional.normalize(q)
    best = []
    for part in q.split(256):
        dot = part @ x.T
        if case["space"] == "l2":
            d = (part * part).sum(1)[:, None] + (x * x).sum(1) - 2 * dot
        else:
            d = 1 - dot if case["space"] == "cosinesimil" else -dot
        best.append(d.topk(case["k"], largest=False).values)
    return None, torch.cat(best).cpu().numpy(), None


def work(case):
    """What a pass cannot do without. A search reads the rows it measures and the lists it walks; how
    many of each follows from efSearch and n (a power law through the engine's own counts on these
    graphs, within a quarter)."""
    n, dim, m, nq = case["n"], case["dim"], case["m"], case["nq"]
    row = dim + 4 if case["space"] == SIFT else 4 * dim
    if case["call"] == "exact":
        return {"bytes": float(n * row + nq * (row + 8 * case["k"])), "flops": 2.0 * nq * n * dim}
    ef = case["ef"]
    if case["call"] == "mixed":
        ef = (64 + case["ef"]) / 2
    if case["call"] == "serve":
        sizes, _, efs = _requests(case)
        nq, ef = sum(sizes), sum(s * e for s, e in zip(sizes, efs)) / sum(sizes)
    walks = max(ef, case["k"]) + 15
    rows = min(0.5 * n, 320 * walks ** 0.277 * (n / 1e6) ** 0.128)
    return {"bytes": nq * (rows * row + walks * 4 * (1 + 1.3 * m) + row + 8 * case["k"]), "flops": 2.0 * nq * rows * dim}
