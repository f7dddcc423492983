"""Timed cases of the engine: what its users run, through the public binding.

A case is a dict of plain values; `listed()` gives the fixed ones, `draw(rng)`
one more of the same ranges.  `prepare(case, seed)` makes what a program holds
before the call (graphs are generated on the GPU from the seed), `run(state)`
is one pass, `work(case)` the bytes a pass cannot do without and
`exact(case, seed)` the same outputs from plain numpy for the small graphs.

Graphs: directed Erdos-Renyi ("er") and R-MAT ("rmat": a=0.57 b=0.19 c=0.19
d=0.05, labels permuted, self-loops and duplicates dropped) of `n` vertices
and `ef` edge draws per vertex.  An R-MAT of an n that is no power of two
keeps the edges between the first n labels of the next power of two.

Kinds:
  decompose  all rows of a graph that stays on the device, again and again
  first      device edge arrays -> new handle -> all rows in device memory
  host       host edge arrays -> new handle -> all rows back in host memory
  text       a text graph file -> new handle -> a .decompCPU file
  maintain   a stream of update batches on a decomposed graph, rows read, then
             the inverse stream (the graph is as before), rows read again
  serve      update requests to several graphs through the serving loop, every
             graph's result read, then the inverse requests
"""
import math
import os
import sys
import tempfile

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (ROOT, os.path.join(ROOT, "d-core-cuda_b200")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

import dcore_b200 as dc  # noqa: E402


def listed():
    return [
        # a small graph kept on the device: launches and host round trips count
        {"name": "er_1k", "kind": "decompose", "graph": "er", "n": 1003, "ef": 8},
        # the reference's plain configuration: ER, 10,000 vertices, 100,000 edges
        {"name": "er_10k", "kind": "first", "graph": "er", "n": 10000, "ef": 10},
        # an ordinary skewed graph of a ragged size (rows are not 16-byte aligned)
        {"name": "rmat_100k_ragged", "kind": "first", "graph": "rmat", "n": 100003, "ef": 16},
        # a large graph at the engine's default launch shapes (one launch for all rows)
        {"name": "rmat20", "kind": "first", "graph": "rmat", "n": 1 << 20, "ef": 16},
        # the headline graph, with launch shapes and row cuts as its autotuner sets them
        {"name": "rmat22_tuned", "kind": "first", "graph": "rmat", "n": 1 << 22, "ef": 16, "tuned": True},
        # host arrays in, host rows out: what a C++ caller of the drop-in ABI does
        {"name": "rmat18_host", "kind": "host", "graph": "rmat", "n": 1 << 18, "ef": 16},
        # the reference's file workflow
        {"name": "rmat15_text", "kind": "text", "graph": "rmat", "n": 1 << 15, "ef": 16},
        # single updates, one call each: maintenance latency
        {"name": "maint_1", "kind": "maintain", "graph": "rmat", "n": 1 << 20, "ef": 16, "batches": 8, "size": 1,
         "insert": 0.5, "hot": False},
        # small batches
        {"name": "maint_100", "kind": "maintain", "graph": "rmat", "n": 1 << 20, "ef": 16, "batches": 2, "size": 100,
         "insert": 0.5, "hot": False},
        # ordinary batches on the headline graph
        {"name": "maint_10k", "kind": "maintain", "graph": "rmat", "n": 1 << 22, "ef": 16, "batches": 1,
         "size": 10000, "insert": 0.5, "hot": False},
        # bulk batches: a quarter of a million updates in one call
        {"name": "maint_250k", "kind": "maintain", "graph": "rmat", "n": 1 << 22, "ef": 16, "batches": 1,
         "size": 250000, "insert": 0.5, "hot": False},
        # the serving loop over graphs of mixed sizes (scales 12..16, edge factors 8..32)
        {"name": "serve_8", "kind": "serve", "graphs": 8, "lo": 12, "hi": 16, "requests": 48, "size": 3000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decompose", "first", "first", "host", "text", "maintain", "maintain", "maintain", "serve"])
    if kind == "serve":
        lo = rng.randint(11, 13)
        return {"kind": kind, "graphs": rng.randint(2, 10), "lo": lo, "hi": rng.randint(lo + 1, 16),
                "requests": rng.randint(8, 64), "size": _log_int(rng, 10, 10000)}
    top = {"decompose": 1 << 21, "first": 1 << 21, "host": 1 << 18, "text": 1 << 15, "maintain": 1 << 21}[kind]
    case = {"kind": kind, "graph": rng.choice(["rmat", "rmat", "er"]), "n": _log_int(rng, 1000, top),
            "ef": rng.randint(4, 24)}
    if rng.random() < 0.3:
        case["n"] = 1 << max(10, int(math.log2(case["n"])))
    if kind in ("decompose", "first") and rng.random() < 0.3:
        case["tuned"] = True
    if kind == "maintain":
        size = _log_int(rng, 1, 100000)
        case.update(size=max(1, min(size, case["n"] // 8)), batches=rng.randint(1, 4),
                    insert=rng.choice([0.0, 0.5, 0.6, 1.0]), hot=rng.random() < 0.2)
    return case


# ---------------------------------------------------------------- inputs
def _keys(graph, n, ef, gen):
    """Sorted distinct edge keys src * n + dst (int64, on the GPU)."""
    m = int(n) * int(ef)
    dev = "cuda"
    if graph == "er":
        k = torch.randint(0, n * (n - 1), (m + m // 16 + 64,), generator=gen, device=dev, dtype=torch.int64)
        src, dst = k // (n - 1), k % (n - 1)
        dst = dst + (dst >= src)
        k = torch.unique(src * n + dst)
        keep = torch.randperm(k.numel(), generator=gen, device=dev)[:m]
        return torch.sort(k[keep])[0]
    scale = max(1, (n - 1).bit_length())
    src = torch.zeros(m, dtype=torch.int64, device=dev)
    dst = torch.zeros(m, dtype=torch.int64, device=dev)
    for _ in range(scale):
        r = torch.rand(m, generator=gen, device=dev)
        src = 2 * src + (r >= 0.76)
        dst = 2 * dst + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    label = torch.randperm(1 << scale, generator=gen, device=dev)
    src, dst = label[src], label[dst]
    ok = (src != dst) & (src < n) & (dst < n)
    return torch.unique(src[ok] * n + dst[ok])


def _split(keys, n):
    return (keys // n).to(torch.int32), (keys % n).to(torch.int32)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _host(t):
    return t.cpu().numpy().astype(np.uint32)


def _updates(keys, n, count, insert, hot, gen):
    """`count` updates with distinct edges, valid in any order: (src, dst,
    is_delete) host arrays.  hot: sources among the top 1 % by out-degree."""
    n_ins = int(round(count * insert))
    n_del = min(count - n_ins, keys.numel() // 2)
    dev = keys.device
    if hot:
        deg = torch.bincount(keys // n, minlength=n)
        top = torch.topk(deg, max(1, n // 100)).indices
        is_top = torch.zeros(n, dtype=torch.bool, device=dev)
        is_top[top] = True
        pool = torch.nonzero(is_top[keys // n]).flatten()
    else:
        pool = None
    total = keys.numel() if pool is None else pool.numel()
    pick = torch.unique(torch.randint(0, total, (4 * n_del + 16,), generator=gen, device=dev))
    pick = pick[torch.randperm(pick.numel(), generator=gen, device=dev)[:n_del]]
    dels = keys[pick if pool is None else pool[pick]]
    u = torch.randint(0, n, (4 * n_ins + 64,), generator=gen, device=dev)
    if hot:
        u = top[u % top.numel()]
    v = torch.randint(0, n, (4 * n_ins + 64,), generator=gen, device=dev)
    k = torch.unique((u * n + v)[u != v])
    at = torch.searchsorted(keys, k).clamp(max=keys.numel() - 1)
    k = k[keys[at] != k]
    ins = k[torch.randperm(k.numel(), generator=gen, device=dev)[:n_ins]]
    both = torch.cat([dels, ins])
    flag = torch.cat([torch.ones_like(dels), torch.zeros_like(ins)])
    order = torch.randperm(both.numel(), generator=gen, device=dev)
    both, flag = both[order], flag[order]
    src, dst = _split(both, n)
    return _host(src), _host(dst), flag.cpu().numpy().astype(np.uint8)


def _pinned(shape):
    return torch.zeros(shape, dtype=torch.int32, pin_memory=True)


def _kmax_about(graph, n, ef):
    """Typical largest kmax of a case's graph (592 at R-MAT 22, edge factor 16)."""
    if graph == "er":
        return max(1, int(0.62 * ef))
    return max(1, int(592 * 1.27 ** (math.log2(n) - 22) * ef / 16))


def _room(graph, n, ef):
    """Rows a program keeps room for: rows above the largest kmax are zero, so
    a buffer of this many rows holds the whole table of any seed's graph."""
    return int(1.35 * _kmax_about(graph, n, ef)) + 16


def _tune(g, case):
    if case.get("tuned"):
        g.set_tuning(peel_blocks_per_sm=3, rows_blocks_per_sm=2, peel_chunk=64, rows_split_permille=(150, 300, 600))
    return g


def prepare(case, seed):
    if case["kind"] == "serve":
        return _prepare_serve(case, seed)
    gen, n, kind = _gen(seed), case["n"], case["kind"]
    keys = _keys(case["graph"], n, case["ef"], gen)
    src, dst = _split(keys, n)
    room = _room(case["graph"], n, case["ef"])
    st = {"case": case, "n": n, "E": keys.numel(), "kmaxes": _pinned(n)}
    if kind == "text":
        st["dir"] = tempfile.TemporaryDirectory()
        st["path"] = os.path.join(st["dir"].name, "graph")
        with open(st["path"], "w") as f:
            f.write("# %d\n" % n)
            f.write("\n".join(map("%d %d".__mod__, zip(src.tolist(), dst.tolist()))))
            f.write("\n")
        st["file"] = np.zeros(8 * n * room, np.uint8)
        return st
    torch.cuda.synchronize()
    g = _tune(dc.Graph.from_device_edges(n, st["E"], src.data_ptr(), dst.data_ptr(), device=0), case)
    g.decompose()
    if kind == "host":
        st["src"], st["dst"] = _host(src), _host(dst)
        st["rows"] = _pinned((room, n))
        g.free()
        return st
    st["rows"] = torch.zeros((room, n), dtype=torch.int32, device="cuda")
    if kind == "first":
        st["src"], st["dst"] = src, dst
        g.free()
        return st
    st["g"] = g
    if kind == "maintain":
        s, d, x = _updates(keys, n, case["batches"] * case["size"], case["insert"], case["hot"], gen)
        size = max(1, -(-len(s) // case["batches"]))
        st["batches"] = [(s[i:i + size], d[i:i + size], x[i:i + size]) for i in range(0, len(s), size)]
        st["inverse"] = [(b[0][::-1].copy(), b[1][::-1].copy(), 1 - b[2][::-1]) for b in st["batches"][::-1]]
        st["rows2"] = torch.zeros((room, n), dtype=torch.int32, device="cuda")
        st["kmaxes2"] = _pinned(n)
    return st


def _prepare_serve(case, seed):
    gen = _gen(seed)
    st = {"case": case, "server": dc.Server(32 << 30, max_concurrent=4), "V": [], "requests": [], "inverse": [],
          "kmaxes": [], "rows": []}
    rng = np.random.default_rng(seed)
    per = [case["requests"] // case["graphs"] + (i < case["requests"] % case["graphs"]) for i in range(case["graphs"])]
    for i in range(case["graphs"]):
        n = 1 << (case["lo"] + i % (case["hi"] - case["lo"] + 1))
        keys = _keys("rmat", n, int(rng.integers(8, 33)), gen)
        src, dst = _split(keys, n)
        gid = st["server"].add_graph(n, _host(src), _host(dst))
        st["V"].append(n)
        st["kmaxes"].append(np.zeros(n, np.int32))
        st["rows"].append(np.zeros((_room("rmat", n, 32), n), np.int32))
        sizes = np.exp(rng.uniform(0, math.log(case["size"]), per[i])).round().astype(int).clip(1)
        sizes = np.minimum(sizes, max(1, keys.numel() // (8 * max(1, per[i]))))
        s, d, x = _updates(keys, n, int(sizes.sum()), 0.6, False, gen)
        o = 0
        for z in sizes:
            if o < len(s):
                st["requests"].append((gid, s[o:o + z], d[o:o + z], x[o:o + z]))
            o += z
        st["server"].result(gid, n, rows=False)  # resident and decomposed
    rng.shuffle(st["requests"])
    st["inverse"] = [(g, s, d, 1 - x) for g, s, d, x in st["requests"][::-1]]
    return st


# ---------------------------------------------------------------- one pass
def _read(st, g, K, rows="rows", kmaxes="kmaxes"):
    """All rows into the program's device buffer and kmax of every vertex into
    its host buffer."""
    if K >= len(st[rows]):
        raise RuntimeError("kmax %d outgrew the row buffer" % K)
    g.rows_to_device(0, K + 1, st[rows].data_ptr())
    g.kmaxes(out=st[kmaxes].numpy())
    g.synchronize()
    return {"rows": st[rows], "kmaxes": st[kmaxes]}


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "decompose":
        K, L = st["g"].decompose()
        return {"kmax": K, "lmax": L, **_read(st, st["g"], K)}
    if kind == "first":
        with dc.Graph.from_device_edges(st["n"], st["E"], st["src"].data_ptr(), st["dst"].data_ptr(),
                                        device=0) as g:
            K, L = _tune(g, case).decompose()
            return {"kmax": K, "lmax": L, **_read(st, g, K)}
    if kind == "host":
        with dc.Graph.from_edges(st["n"], st["src"], st["dst"], device=0) as g:
            K, L = g.decompose()
            g.rows(0, K + 1, out=st["rows"].numpy()[:K + 1])
            g.kmaxes(out=st["kmaxes"].numpy())
            return {"kmax": K, "lmax": L, "rows": st["rows"], "kmaxes": st["kmaxes"]}
    if kind == "text":
        with dc.Graph.load_text_device(st["path"], device=0) as g:
            K, L = g.decompose()
            out = st["path"] + ".decompCPU"
            g.write_decomp_cpu_device(out)
            with open(out, "rb") as f:
                size = f.readinto(st["file"])
            return {"kmax": K, "lmax": L, "size": size, "file": st["file"]}
    if kind == "maintain":
        g = st["g"]
        for s, d, x in st["batches"]:
            info = g.maintain(s, d, x)
        there = {"kmax": info["kmax"], "lmax": info["lmax"], **_read(st, g, info["kmax"])}
        for s, d, x in st["inverse"]:
            info = g.maintain(s, d, x)
        back = {"kmax": info["kmax"], "lmax": info["lmax"], **_read(st, g, info["kmax"], "rows2", "kmaxes2")}
        return {"there": there, "back": back}
    sv = st["server"]
    for gid, s, d, x in st["requests"]:
        sv.submit(gid, s, d, x)
    sv.drain()
    for gid, V in enumerate(st["V"]):
        kmaxes, rows = sv.result(gid, V)
        st["kmaxes"][gid][:], st["rows"][gid][:len(rows)] = kmaxes, rows
    for gid, s, d, x in st["inverse"]:
        sv.submit(gid, s, d, x)
    sv.drain()
    sv.completions()
    return {"kmaxes": st["kmaxes"], "rows": st["rows"]}


# ---------------------------------------------------------------- the least a pass moves
def work(case):
    """Every input read once and every output written once: the edges (8
    bytes each, or the two adjacency sides of a graph that is kept), the dense
    rows and kmax; for maintenance the updates, and the rows read twice."""
    if case["kind"] == "serve":
        b = 0
        for i in range(case["graphs"]):
            n = 1 << (case["lo"] + i % (case["hi"] - case["lo"] + 1))
            b += 4 * n * (_kmax_about("rmat", n, 20) + 2)
        return {"bytes": b + 2 * 9 * case["requests"] * case["size"] / max(1.0, math.log(case["size"])), "flops": 0}
    n, ef = case["n"], case["ef"]
    rows = 4 * n * (_kmax_about(case["graph"], n, ef) + 2)
    if case["kind"] == "maintain":
        return {"bytes": 2 * rows + 2 * 9 * case["batches"] * case["size"], "flops": 0}
    return {"bytes": 8 * n * ef + rows, "flops": 0}


# ---------------------------------------------------------------- the same outputs, plainly
def _plain(n, src, dst):
    """kmax of every vertex and every row by definition: row k of v is the
    largest l with v in the subgraph of in-degrees >= k and out-degrees >= l."""
    def shrink(alive, k, l):
        while True:
            e = alive[src] & alive[dst]
            bad = alive & ((np.bincount(dst[e], minlength=n) < k) | (np.bincount(src[e], minlength=n) < l))
            if not bad.any():
                return alive
            alive = alive & ~bad
    kmaxes = np.zeros(n, np.int64)
    rows, alive, k = [], np.ones(n, bool), 0
    while True:
        alive = shrink(alive, k, 0)
        if not alive.any():
            return kmaxes, np.stack(rows)
        kmaxes[alive] = k
        row, inner, l = np.zeros(n, np.int64), alive, 0
        while inner.any():
            row[inner] = l
            l += 1
            inner = shrink(inner, k, l)
        rows.append(row)
        k += 1


def exact(case, seed):
    if case["kind"] not in ("decompose", "first", "host") or case["n"] * case["ef"] > 300000:
        return None
    n = case["n"]
    src, dst = (t.cpu().numpy().astype(np.int64) for t in _split(_keys(case["graph"], n, case["ef"], _gen(seed)), n))
    kmaxes, rows = _plain(n, src, dst)
    table = np.zeros((_room(case["graph"], n, case["ef"]), n), np.int64)
    table[:len(rows)] = rows
    return {"kmax": len(rows) - 1, "lmax": int(rows[0].max()), "rows": table, "kmaxes": kmaxes}
