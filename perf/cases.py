"""The work that a program has this library do, as cases that can be timed.

Three kinds of program use the library: one that asks a resident index for
distances (one pair, a device batch, a host batch, a stream of requests through
the server), one that builds an index from a road graph's files, and one that
keeps many graphs and rebuilds them when arc weights change.  Every case makes
its own seeded road graph in the Edge / ID / Cut formats and goes through the
package's public calls.

A built index stays on the GPU behind its handle and is read through queries,
so a build returns the elimination order, the tree and the distances from a
few sources to every vertex; the smallest build returns every label entry.
"""
import math
import os
import random
import sys
import tempfile

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "gpu-h2h_gb300"))

import gpuh2h  # noqa: E402

C_HEIGHT = 2        # ChangeToGlobalHeight of every workload of the benchmark
THREADS = os.cpu_count() or 4
LOCAL_HOPS = 20     # "local" pairs lie within a 20-hop walk of each other
SOURCES = 4         # a build is read back as distances from this many sources to every vertex


def listed():
    return [
        # an interactive lookup: one distance at a time
        dict(name="one_pair", kind="pair", n=4096),
        # a route service's small batch, pairs already on the device
        dict(name="batch_1k", kind="device", n=20000, uniform=1000, local=0, lca=True),
        # a matrix request: the batch size whose p50 / p99 the benchmark quotes
        dict(name="batch_100k", kind="device", n=264346, uniform=100000, local=0, lca=True),
        # the benchmark's step: a million uniform and a million local pairs
        dict(name="batch_2m", kind="device", n=264346, uniform=1000000, local=1000000, lca=True),
        # the other query mode (every common ancestor instead of the LCA's separator), odd batch size
        dict(name="batch_nolca", kind="device", n=70000, uniform=60000, local=39991, lca=False),
        # pairs and answers in page-locked host memory, copies included
        dict(name="host_2m", kind="host", n=70000, uniform=1000000, local=1000000, lca=True),
        # mixed request sizes on two resident graphs through the query server
        dict(name="server_mix", kind="server", n=20000, n2=70000, requests=48, size_hi=100000),
        # the smallest build: a town (the 64 x 64 grid of the tests), labels read back whole
        dict(name="build_4k", kind="labels", n=4096),
        # a city (the vertex count of the New York road graph) from its files to answers
        dict(name="build_264k", kind="build", n=264346),
        # a state: a tree deeper than 2,048 levels
        dict(name="build_1m", kind="build", n=1000000),
        # many small regions built in one go
        dict(name="batch_build", kind="batch", graphs=16, n=2000, n_hi=40000),
        # the same regions after a traffic update: new weights on every arc
        dict(name="batch_rebuild", kind="rebuild", graphs=16, n=2000, n_hi=40000),
    ]


def draw(rng):
    def logu(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["pair", "device", "device", "device", "host", "server", "labels", "build", "build", "build",
                       "batch", "rebuild"])
    if kind == "pair":
        return dict(kind=kind, n=logu(500, 70000))
    if kind in ("device", "host"):
        pairs = logu(100, 2000000)
        local = int(pairs * rng.choice([0.0, 0.5, rng.random()]))
        return dict(kind=kind, n=logu(2000, 264346), uniform=pairs - local, local=local, lca=rng.random() < 0.75)
    if kind == "server":
        return dict(kind=kind, n=logu(2000, 70000), n2=logu(2000, 70000), requests=logu(8, 64),
                    size_hi=logu(100, 100000))
    if kind == "labels":
        return dict(kind=kind, n=logu(200, 6000))
    if kind == "build":
        return dict(kind=kind, n=logu(6000, 700000))
    return dict(kind=kind, graphs=logu(2, 16), n=logu(500, 2000), n_hi=logu(4000, 40000))


# ---- inputs

def _road(root, name, n, rng):
    """One road graph of the benchmark's shape: a jittered grid with diagonals
    and a highway layer, 2.776 arcs per vertex, latitude / longitude
    partition.  Returns its files and the partition's height."""
    height = max(2, math.ceil(math.log2(n / 256)))
    gpuh2h.generate_road(root, name, n=n, target_arcs=int(round(n * 733846 / 264346)),
                         aspect_milli=rng.choice([1000, 1300, 1500]), jitter_milli=300, diag_permille=50, hw_tiers=1,
                         hw_permille10=50, hw_k=3, hw_scale_milli=400, partition_height=height,
                         seed=rng.randrange(1, 1 << 30), cols=0, drop_permille=0)
    return gpuh2h.files_for(root, name), height


def _build(files, height):
    g = gpuh2h.Graph("g", height, C_HEIGHT, THREADS, 1, files=files)
    g.contraction_noHub(1)
    g.constructLabel_noHub(2, 1, gpuh2h.LABEL_L4)
    return g


def _pairs(g, n, uniform, local, seed):
    x, y = gpuh2h.uniform_pairs(n, uniform, seed)
    if local:
        lx, ly = g.local_pairs(local, LOCAL_HOPS, seed + 1)
        x, y = np.concatenate([x, lx]), np.concatenate([y, ly])
    return x, y


def _source_pairs(n, rng):
    """Pairs (s, v) of SOURCES random sources and every vertex v."""
    src = np.array([rng.randrange(n) for _ in range(SOURCES)], np.int32)
    return np.repeat(src, n), np.tile(np.arange(n, dtype=np.int32), SOURCES)


def _log_uniform(lo, hi, count, key):
    """`count` sizes log-uniform in [lo, hi], the same for every seed."""
    rng = random.Random(key)
    return [int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) for _ in range(count)]


def _files(case, seed):
    """The case's road graphs on disk: (keep-alive folder, [(files, height, n)], rng)."""
    rng = random.Random(seed)
    tmp = tempfile.TemporaryDirectory(prefix="cases_")
    kind, n = case["kind"], case["n"]
    if kind == "labels":
        # how many entries the labels hold depends on which roads there are, so
        # the roads are the case's and the weights the seed's
        files, height = _road(tmp.name, "g0", n, random.Random(n))
        with gpuh2h.Graph("g", height, C_HEIGHT, THREADS, 1, files=files) as g:
            off, v, w = g.input_arcs()
        gpuh2h.write_edge_file(files[0], off, v, _new_weights(w, off, v, seed))
        return tmp, [(files, height, n)], rng
    sizes = _log_uniform(n, case["n_hi"], case["graphs"], n) if kind in ("batch", "rebuild") else \
        [n, case["n2"]] if kind == "server" else [n]
    graphs = []
    for i, n in enumerate(sizes):
        files, height = _road(tmp.name, "g%d" % i, n, rng)
        graphs.append((files, height, n))
    return tmp, graphs, rng


def _new_weights(w, off, v, seed):
    """Symmetric new weights: up to twice the old one, the same both ways."""
    src = np.repeat(np.arange(len(off) - 1, dtype=np.int64), np.diff(off))
    lo, hi = np.minimum(src, v), np.maximum(src, v)
    return (w + (lo * 31 + hi * 17 + seed) % (w.astype(np.int64) + 1)).astype(np.int32)


def _dev(a):
    return torch.from_numpy(a).cuda()


def prepare(case, seed):
    tmp, graphs, rng = _files(case, seed)
    kind = case["kind"]
    st = dict(kind=kind, tmp=tmp, graphs=graphs)
    qseed = rng.randrange(1, 1 << 30)
    if kind in ("pair", "device", "host"):
        files, height, n = graphs[0]
        g = st["g"] = _build(files, height)
        st["mode"] = gpuh2h.QUERY_LCA if case.get("lca", True) else gpuh2h.QUERY_NOLCA
        if kind == "pair":
            x, y = gpuh2h.uniform_pairs(n, 1, qseed)
            st["x"], st["y"] = int(x[0]), int(y[0])
            return st
        x, y = _pairs(g, n, case["uniform"], case["local"], qseed)
        if kind == "device":
            st["x"], st["y"] = _dev(x), _dev(y)
            st["out"] = torch.empty_like(st["x"])
        else:
            st["x"], st["y"] = torch.from_numpy(x).pin_memory(), torch.from_numpy(y).pin_memory()
            st["out"] = torch.empty_like(st["x"]).pin_memory()
    elif kind == "server":
        st["g"] = [_build(files, height) for files, height, _ in graphs]
        st["srv"] = gpuh2h.Server(slots=4, slot_pairs=1 << 17)
        ids = [st["srv"].add(g) for g in st["g"]]
        st["req"] = []
        for k, size in enumerate(_log_uniform(1, case["size_hi"], case["requests"], case["n"])):
            i = k % 2
            x, y = gpuh2h.uniform_pairs(graphs[i][2], size, qseed + k)
            pin = [torch.from_numpy(a).pin_memory() for a in (x, y, np.empty(size, np.int32))]
            st["req"].append((ids[i], pin, [t.numpy() for t in pin]))
    else:
        st["pairs"] = []
        for _, _, n in graphs:
            x, y = _source_pairs(n, rng)
            st["pairs"].append((_dev(x), _dev(y)))
        if kind == "rebuild":
            st["g"] = [gpuh2h.Graph("g", h, C_HEIGHT, THREADS, 1, files=f) for f, h, _ in graphs]
            st["batch"] = gpuh2h.Batch(st["g"], THREADS)
            st["w"] = []
            for g in st["g"]:
                off, v, w = g.input_arcs()
                st["w"].append(_new_weights(w, off, v, seed))
    return st


# ---- one pass

def _answers(g, pairs, mode=gpuh2h.QUERY_LCA):
    x, y = pairs
    out = torch.empty_like(x)
    g.query_device(x.data_ptr(), y.data_ptr(), out.data_ptr(), len(x), mode, torch.cuda.current_stream().cuda_stream)
    return out


def run(state):
    kind = state["kind"]
    if kind == "pair":
        return state["g"].H2HDistancQuery_UsingLCA_noHub(state["x"], state["y"])
    if kind == "device":
        x, y, out = state["x"], state["y"], state["out"]
        state["g"].query_device(x.data_ptr(), y.data_ptr(), out.data_ptr(), len(x), state["mode"],
                                torch.cuda.current_stream().cuda_stream)
        return out
    if kind == "host":
        x, y, out = state["x"], state["y"], state["out"]
        state["g"].query_host_ptr(x.data_ptr(), y.data_ptr(), out.data_ptr(), len(x), state["mode"])
        return out
    if kind == "server":
        srv = state["srv"]
        ids = [srv.submit(gid, *arrays) for gid, _, arrays in state["req"]]
        for r in ids:
            srv.wait(r)
            srv.release(r)
        return [pin[2] for _, pin, _ in state["req"]]
    if kind == "labels":
        files, height, _ = state["graphs"][0]
        with _build(files, height) as g:
            father, depth, _ = g.tree()
            return dict(g.labels(), order=g.order(), father=father, depth=depth)
    if kind == "build":
        files, height, _ = state["graphs"][0]
        with _build(files, height) as g:
            father, depth, _ = g.tree()
            return dict(distances=_answers(g, state["pairs"][0]), order=g.order(), father=father, depth=depth)
    if kind == "batch":
        gs = [gpuh2h.Graph("g", h, C_HEIGHT, THREADS, 1, files=f) for f, h, _ in state["graphs"]]
        b = gpuh2h.Batch(gs, THREADS)
        out = dict(distances=[_answers(g, p) for g, p in zip(gs, state["pairs"])], order=[g.order() for g in gs])
        b.close()
        for g in gs:
            g.close()
        return out
    for i, w in enumerate(state["w"]):
        state["batch"].set_weights(i, w)
    state["batch"].rebuild()
    return [_answers(g, p) for g, p in zip(state["g"], state["pairs"])]


# ---- what a pass cannot do without

def _label_entries(n):
    # one entry per vertex and ancestor; road graphs' trees average about
    # 2 sqrt(n) ancestors (264k vertices: 304M entries, 6.26M: 28.7e9)
    return 2.0 * n ** 1.5


def _build_work(n):
    # the arcs once (two ids and a weight) and every label entry once; about
    # 14.5 min-plus updates of two operations per label entry
    return 12 * 2.776 * n + 4 * _label_entries(n), 29 * _label_entries(n)


def _pair_bytes(n, lca):
    # ids, answer and LCA lookup; then two label entries per position of the
    # LCA's separator (about sqrt(n) / 3, with 4 bytes for the position) or
    # per common ancestor (about 0.4 sqrt(n): uniform pairs meet near the top)
    return 84 + 12 * math.sqrt(n) / 3 if lca else 68 + 8 * 0.4 * math.sqrt(n)


def work(case):
    kind, n = case["kind"], case["n"]
    if kind == "pair":
        return dict(bytes=_pair_bytes(n, True), flops=2 * math.sqrt(n) / 3)
    if kind in ("device", "host"):
        q = case["uniform"] + case["local"]
        return dict(bytes=q * _pair_bytes(n, case["lca"]), flops=q * 2 * math.sqrt(n) / 3)
    if kind == "server":
        mean = (case["size_hi"] - 1) / max(math.log(case["size_hi"]), 1.0)  # of the log-uniform sizes
        per = (_pair_bytes(n, True) + _pair_bytes(case["n2"], True)) / 2
        return dict(bytes=case["requests"] * mean * per, flops=case["requests"] * mean * 2 * math.sqrt(n) / 3)
    if kind in ("labels", "build"):
        b, f = _build_work(n)
        if kind == "build":
            b += SOURCES * n * _pair_bytes(n, True)
        return dict(bytes=b, flops=f)
    lo, hi, b, f = math.log(n), math.log(case["n_hi"]), 0.0, 0.0
    for i in range(case["graphs"]):
        k = math.exp(lo + (hi - lo) * (i + 0.5) / case["graphs"])
        gb, gf = _build_work(k)
        b += gb + SOURCES * k * _pair_bytes(k, True)
        f += gf
    return dict(bytes=b, flops=f)


# ---- the exact distances, by plain relaxation in 64 bits

def _arcs(files):
    """(n, tail, head, weight) of an Edge file, self loops dropped."""
    with open(files[0]) as f:
        n = int(f.readline().split()[0])
        a = np.array(f.read().replace("a", " ").split(), np.int64).reshape(-1, 3)
    a = a[a[:, 0] != a[:, 1]]
    return n, a[:, 0] - 1, a[:, 1] - 1, a[:, 2]


def _neighbours(n, u, v, w):
    """Padded neighbour and weight tables, one column per arc of a vertex."""
    o = np.argsort(u, kind="stable")
    u, v, w = u[o], v[o], w[o]
    slot = np.arange(len(u)) - np.searchsorted(u, u)
    width = int(slot.max()) + 1
    nb = np.repeat(np.arange(n)[:, None], width, 1)
    wt = np.zeros((n, width), np.int64)
    wt[:] = 1 << 40
    nb[u, slot], wt[u, slot] = v, w
    return torch.from_numpy(nb).cuda(), torch.from_numpy(wt).cuda()


def _distances(tables, n, sources):
    """Distances from each source to every vertex, by relaxing all arcs until nothing changes."""
    nb, wt = tables
    d = torch.full((len(sources), n), 1 << 40, dtype=torch.int64, device="cuda")
    d[torch.arange(len(sources)), torch.as_tensor(sources)] = 0
    while True:
        before = d
        for _ in range(32):
            step = d
            for k in range(nb.shape[1]):
                step = torch.minimum(step, d[:, nb[:, k]] + wt[:, k])
            d = step
        if torch.equal(before, d):
            return d


def exact(case, seed):
    kind = case["kind"]
    if kind in ("host", "server") or (kind == "device" and case["uniform"] + case["local"] > 1000):
        return None  # a source per pair: too many searches
    if kind == "labels":
        return None  # which ancestors a row holds is the elimination's choice
    tmp, graphs, rng = _files(case, seed)
    qseed = rng.randrange(1, 1 << 30)
    if kind == "pair":
        n, u, v, w = _arcs(graphs[0][0])
        x, y = gpuh2h.uniform_pairs(n, 1, qseed)
        return int(_distances(_neighbours(n, u, v, w), n, [int(x[0])])[0, int(y[0])])
    if kind == "device":
        if case["local"]:
            return None  # local pairs are drawn from the loaded graph
        n, u, v, w = _arcs(graphs[0][0])
        x, y = gpuh2h.uniform_pairs(n, case["uniform"], qseed)
        d = _distances(_neighbours(n, u, v, w), n, x.astype(np.int64))
        return d[torch.arange(len(x)), torch.from_numpy(y.astype(np.int64))]
    res = []
    for files, _, n in graphs:
        _, u, v, w = _arcs(files)
        if kind == "rebuild":
            lo, hi = np.minimum(u, v), np.maximum(u, v)
            w = w + (lo * 31 + hi * 17 + seed) % (w + 1)
        sources = [rng.randrange(n) for _ in range(SOURCES)]
        res.append(_distances(_neighbours(n, u, v, w), n, sources).reshape(-1))
    if kind == "rebuild":
        return res
    if kind == "batch":
        return dict(distances=res, order=[None] * len(res))
    return dict(distances=res[0], order=None, father=None, depth=None)
