"""The work that is timed: what a user of the update path has it do.

A case names a workload generator of this package with its sizes and options.
`prepare` builds what a program holds before the call (device graphs, a
snapshot of them, the update batches); `run` makes one pass through the public
entry points and returns what they return.  A pass starts from the snapshot
(`Graph.copy_from`), so it can be repeated.  Results whose number depends on the
data (recovered edges, a graph's slots) are written to buffers of a fixed size,
as a program that calls the C interface does.

Kinds of work:
  update   one graph: a stream of insertions, then a stream of deletions
           (either may be empty), on a 2-D grid or a 3-D mesh
  files    mixed insert / delete stream files on an R-MAT graph (hub rows)
  many     the insertion streams of many graphs, one launch per round
  serve    requests for many resident graphs, all pending at once
  session  what the command-line updaters do between reading and writing
           their files: build both graphs from edge lists, apply the
           insertions and the deletions, export both graphs
"""
from __future__ import annotations

import math

import numpy as np
import torch

import dygrass_b200 as D
from dygrass_b200 import multi, serve, workloads

UNIFORM, WEIGHTED = D.TRANSITION_UNIFORM, D.TRANSITION_WEIGHTED


def _update(name, dims, ins, dels, batch=0, walkers=512, steps=100, threshold=100.0, transition=UNIFORM,
            with_g=True, device=False):
    return {"name": name, "kind": "update", "nx": dims[0], "ny": dims[1], "nz": dims[2], "ins": ins,
            "dels": dels, "batch": batch, "walkers": walkers, "steps": steps, "threshold": threshold,
            "transition": transition, "with_g": with_g, "device": device}


def _files(name, scale, files, size, walkers=256, steps=128, threshold=50.0, transition=UNIFORM):
    return {"name": name, "kind": "files", "scale": scale, "files": files, "size": size, "walkers": walkers,
            "steps": steps, "threshold": threshold, "transition": transition}


def listed():
    return [
        # an interactive edit: a few edges of a small graph, one batch from host arrays; latency is all
        _update("grid_insert_32", (100, 100, 1), 32, 0, batch=32, steps=64, threshold=10.0, with_g=False),
        # the same for a few deletions, with their recovery
        _update("mesh_delete_64", (20, 20, 20), 0, 64, batch=64),
        # the reference's small workload: 1,000 insertions in its ten batches, from host arrays
        _update("grid_stream_1000", (100, 100, 1), 1000, 0, steps=64, threshold=10.0, with_g=False),
        # an ordinary graph of odd sizes, ragged batches and a walker count that is no power of two
        _update("mesh_mixed_odd", (37, 41, 29), 4999, 7777, batch=1013, walkers=160, steps=77),
        # the headline workload's insertions at full size, arrays resident on the device
        _update("mesh_insert_200k", (100, 100, 100), 200_000, 0, device=True),
        # the headline workload's deletions at full size
        _update("mesh_delete_297k", (100, 100, 100), 0, 297_000, device=True),
        # the weight-proportional transition, both directions
        _update("mesh_weighted", (40, 40, 40), 8000, 12000, transition=WEIGHTED, device=True),
        # a power-law graph fed by stream files of the reference's usual size, rows of thousands of slots
        _files("rmat_files", 16, 12, 4096),
        # the same with weight-proportional walks through the hub rows
        _files("rmat_weighted", 13, 6, 1000, transition=WEIGHTED),
        # a fleet of uneven graphs updated together
        {"name": "many_graphs", "kind": "many", "graphs": 24, "n_lo": 1000, "n_hi": 60_000, "walkers": 512,
         "steps": 100, "threshold": 100.0},
        # a server at saturation: small and large requests for resident graphs of all three generators
        {"name": "serve_saturated", "kind": "serve", "graphs": 12, "requests": 150, "size_hi": 4096},
        # a whole command-line run without its file reading and writing
        {"name": "session_mesh", "kind": "session", "nx": 48, "ny": 48, "nz": 48, "ins": 20_000, "dels": 30_000,
         "walkers": 512, "steps": 100, "threshold": 100.0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _walk_options(rng):
    return {"walkers": 32 * rng.choice([1, 2, 3, 5, 8, 16, 16, 16, 32]), "steps": rng.choice([20, 50, 64, 100, 100, 128]),
            "threshold": float(rng.choice([10, 50, 100, 100, 200]))}


def draw(rng):
    kind = rng.choice(["update"] * 5 + ["files"] * 2 + ["many", "serve", "session"])
    opt = _walk_options(rng)
    weighted = WEIGHTED if rng.random() < 0.2 else UNIFORM
    if kind == "update":
        flat = rng.random() < 0.3
        top = 250 if flat else (36 if weighted else 62)
        dims = [_log(rng, 16 if flat else 8, top) for _ in range(2 if flat else 3)] + [1] * flat
        n = dims[0] * dims[1] * dims[2]
        most = max(4, min(n // 5, 20_000 if weighted else 60_000))
        way = rng.choice(["ins", "dels", "both"])
        ins = _log(rng, 8, max(8, most)) if way != "dels" else 0
        dels = _log(rng, 40, max(40, most)) if way != "ins" else 0
        batch = 0 if rng.random() < 0.6 else max(_log(rng, 1, max(ins, dels)), max(ins, dels) // 25 + 1)
        c = _update("", dims, ins, dels, batch=batch, transition=weighted, with_g=dels > 0 or rng.random() < 0.5,
                    device=rng.random() < 0.5)
        del c["name"]
        return {**c, **opt}
    if kind == "files":
        size = _log(rng, 10, 4096)
        c = _files("", rng.randint(9, 13 if weighted else 15), rng.randint(2, 8), size, transition=weighted)
        del c["name"]
        return {**c, **opt}
    if kind == "many":
        lo = _log(rng, 200, 2000)
        return {"kind": kind, "graphs": rng.randint(2, 24), "n_lo": lo, "n_hi": _log(rng, 2 * lo, 40_000), **opt}
    if kind == "serve":
        return {"kind": kind, "graphs": rng.randint(3, 10), "requests": _log(rng, 10, 150), "size_hi": _log(rng, 32, 4096)}
    d = [_log(rng, 10, 48) for _ in range(3)]
    n = d[0] * d[1] * d[2]
    return {"kind": kind, "nx": d[0], "ny": d[1], "nz": d[2], "ins": _log(rng, 10, n // 5), "dels": _log(rng, 40, n // 4), **opt}


# ------------------------------------------------------------------ inputs

def _params(case, seed, insert):
    return D.WalkParams.make(threshold=case["threshold"] if insert else 100.0, walkers=case["walkers"],
                             max_steps=case["steps"], transition=case.get("transition", UNIFORM), seed=seed)


def _lattice(case, seed):
    """The grid or mesh of a case, its sparsifier, insertions and deletions (host arrays), with the weight
    laws of the generators in dygrass_b200.workloads."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if nz == 1:
        law, lo, hi, frac, far = workloads.W_UNIFORM, 0.5, 2.0, 0.10, 8
    else:
        law, lo, hi, frac, far = workloads.W_LOGUNIFORM, 1e-2, 1e2, 0.05, 10
    s, d, w = workloads.lattice(nx, ny, nz, law, lo, hi, seed + 1)
    idx = workloads.sparsifier(nx * ny * nz, s, d, w, frac, seed + 2)
    ins = workloads.lattice_inserts(nx, ny, nz, s, d, case["ins"], 2, far, law, lo, hi, seed + 3)
    gs, gd = np.concatenate([s, ins[0]]), np.concatenate([d, ins[1]])
    di = workloads.sample(len(gs), min(case["dels"], len(gs)), seed + 4) if case["dels"] else np.empty(0, np.int64)
    return {"n": nx * ny * nz, "g": (s, d, w), "h": (s[idx], d[idx], w[idx]), "ins": ins, "dels": (gs[di], gd[di])}


def _on_device(arrays):
    return [torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).cuda() for a in arrays]


SERVED = ("conductance", "found_at", "accepted", "status", "rec_src", "rec_dst", "rec_kind")


def _zeros(*sizes, on_device=False):
    host = tuple(np.zeros(k, t) for k, t in sizes)
    return tuple(_on_device(host)) if on_device else host


def _records(n, on_device=False):
    """Status, conductance and recovered edges (the last three of one size) of n deletions."""
    cap = 64 * n + 4096
    return _zeros((n, np.int32), (n, np.float32), (cap, np.uint32), (cap, np.uint32), (cap, np.uint8), on_device=on_device)


def prepare(case, seed):
    kind = case["kind"]
    seed = 1000 * int(seed) + 17
    st = {"case": case, "kind": kind}
    if kind in ("update", "session"):
        x = _lattice(case, seed)
        st |= {"n": x["n"], "ip": _params(case, seed, True), "dp": _params(case, seed, False), "ins": x["ins"],
               "dels": x["dels"]}
        if kind == "session":
            st |= {"g": x["g"], "h": x["h"]}
            cap = 2 * (len(x["g"][0]) + case["ins"])
            st["rows"] = {k: (np.zeros(x["n"] + 1, np.uint64), np.zeros(cap, np.uint32), np.zeros(cap, np.float32)) for k in "HG"}
        else:
            st["H0"] = D.Graph.from_edges(x["n"], *x["h"])
            st["H"] = st["H0"].clone()
            if case["with_g"]:
                st["G0"] = D.Graph.from_edges(x["n"], *x["g"])
                st["G"] = st["G0"].clone()
        on_device = case.get("device", False)
        if on_device:
            st["ins"], st["dels"] = _on_device(x["ins"]), _on_device(x["dels"])
        ni, nd = len(x["ins"][0]), len(x["dels"][0])
        st["out"] = D.IncrementalResult(*_zeros((ni, np.int32), (ni, np.float32), (ni, np.uint8), on_device=on_device))
        st["rec"] = _records(nd, on_device)
    elif kind == "files":
        wl = workloads.rmat_mixed(scale=case["scale"], n_updates=case["files"] * case["size"], file_size=case["size"],
                                  seed=seed, walkers=case["walkers"], max_steps=case["steps"])
        st |= {"ip": _params(case, seed, True), "dp": _params(case, seed, False), "files": wl.files}
        st["H0"] = D.Graph.from_edges(wl.n, wl.h_src, wl.h_dst, wl.h_w)
        st["G0"] = D.Graph.from_edges(wl.n, wl.g_src, wl.g_dst, wl.g_w)
        st["H"], st["G"] = st["H0"].clone(), st["G0"].clone()
        st["rec"] = [_records(len(f[1])) for f in wl.files]
    elif kind == "many":
        graphs, ip = workloads.rgg_many(case["graphs"], case["n_lo"], case["n_hi"], seed=seed, walkers=case["walkers"],
                                        max_steps=case["steps"], threshold=case["threshold"])
        st["M"] = multi.ManyGraphs(graphs)
        st |= {"ip": ip, "plan": st["M"].plan(), "H0": st["M"].H.clone(), "G0": st["M"].G.clone()}
        k = case["graphs"] * (case["n_hi"] // 20 + 1)
        st["out"] = _zeros((k, np.int32), (k, np.float32), (k, np.uint8))
        ends = np.cumsum([0] + [len(r.src) for r in st["plan"].rounds])
        st["outs"] = [D.IncrementalResult(*(a[i:j] for a in st["out"])) for i, j in zip(ends, ends[1:])]
    else:
        graphs, ip, dp = workloads.serving_mix(case["graphs"], seed=seed)
        st["server"] = serve.Server(graphs, ip, dp)
        st["server"].snapshot()
        st["requests"] = serve.poisson_requests(graphs, 1.0, case["requests"], seed, size_hi=case["size_hi"])
        for r in st["requests"]:
            r.arrival = 0.0
        k = case["requests"] * case["size_hi"]
        st["out"] = dict(zip(SERVED, _zeros((k, np.float32), (k, np.int32), (k, np.uint8), (k, np.int32), (2 * k, np.uint32),
                                            (2 * k, np.uint32), (2 * k, np.uint8))))
    return st


# -------------------------------------------------------------------- pass

def _insert_delete(st, H, G, batch):
    """The insertion stream, then the deletion stream, as plain values."""
    out = {}
    if len(st["ins"][0]):
        r = D.incremental_stream(H, *st["ins"], st["ip"], batch, G=G, out=st["out"])
        out |= {"found_at": r.found_at, "conductance": r.conductance, "accepted": r.accepted}
    if len(st["dels"][0]):
        status, cond, rx, ry, rk = st["rec"]
        n = D.decremental_stream_into(G, H, *st["dels"], st["dp"], status, cond, rx, ry, rk, len(rx), batch)
        out |= {"status": status, "del_conductance": cond, "rec_src": rx, "rec_dst": ry, "rec_kind": rk, "n_rec": n}
    return out


def run(st):
    kind = st["kind"]
    if kind == "update":
        st["H"].copy_from(st["H0"])
        if "G" in st:
            st["G"].copy_from(st["G0"])
        return _insert_delete(st, st["H"], st.get("G"), st["case"]["batch"])
    if kind == "session":
        H, G = D.Graph.from_edges(st["n"], *st["h"]), D.Graph.from_edges(st["n"], *st["g"])
        out = _insert_delete(st, H, G, 0)
        for name, graph in (("H", H), ("G", G)):
            for buf, rows in zip(st["rows"][name], graph.export()):
                buf[:len(rows)] = rows
            graph.close()
        return out | st["rows"]
    if kind == "files":
        st["H"].copy_from(st["H0"])
        st["G"].copy_from(st["G0"])
        counts, at = [], 0
        for (op, src, dst, w), rec in zip(st["files"], st["rec"]):
            counts.append(D.stream_file_into(st["G"], st["H"], op, src, dst, w, st["dp"] if op else st["ip"], *rec,
                                             len(rec[2]), first_update_id=at))
            at += len(src)
        return {"counts": np.array(counts)} | {f: [rec[i] for rec in st["rec"]] for i, f in
                                               enumerate(("status", "conductance", "rec_src", "rec_dst", "rec_kind"))}
    if kind == "many":
        M = st["M"]
        M.H.copy_from(st["H0"])
        M.G.copy_from(st["G0"])
        M.run(st["plan"], st["ip"], outs=st["outs"])
        return st["out"]
    st["server"].restore()
    st["server"].serve(st["requests"])
    for f in SERVED:
        at = 0
        for r in st["requests"]:
            got = getattr(r, f)
            if got is not None:
                st["out"][f][at:at + len(got)] = got
                at += len(got)
    return st["out"]


# -------------------------------------------------------------------- work

def work(case):
    """Batches read and results written once, the graphs restored (read and written once), and for every walker
    that has to start one move: the 16 bytes of a row descriptor and of the slot it takes (about a third of a
    lattice's deleted edges are in the sparsifier and walked)."""
    kind = case["kind"]

    def graph(n, edges):
        return 24 * edges + 12 * n

    def moves(edges):
        return edges * case.get("walkers", 512) * 16

    if kind in ("update", "session"):
        n = case["nx"] * case["ny"] * case["nz"]
        dense, sparse = n * (2 if case["nz"] == 1 else 3), int(1.1 * n)
        b = 21 * case["ins"] + 16 * case["dels"] + moves(case["ins"]) + moves(case["dels"] // 3)
        b += 2 * graph(n, sparse) + (2 * graph(n, dense) if case.get("with_g", True) else 0)
    elif kind == "files":
        n, upd = int(0.62 * 2 ** case["scale"]), case["files"] * case["size"]
        b = 20 * upd + moves(int(0.6 * upd)) + 2 * graph(n, 16 * 2 ** case["scale"]) + 2 * graph(n, int(2.2 * n))
    elif kind == "many":
        lo, hi = case["n_lo"], case["n_hi"]
        n = int(case["graphs"] * (hi - lo) / math.log(hi / lo))
        ins = n // 20
        b = 29 * ins + moves(ins) + 2 * graph(n, 4 * n) + 2 * graph(n, int(1.3 * n))
    else:
        upd = int(case["requests"] * case["size_hi"] / math.log(case["size_hi"] + 1))
        n = case["graphs"] * 30_000
        b = 30 * upd + moves(int(0.65 * upd)) + 2 * graph(n, 6 * n) + 2 * graph(n, int(1.3 * n))
    return {"bytes": b, "flops": 0}


# ------------------------------------------------------------------- exact

def _philox(block, walker, uid, domain, key):
    """Philox4x32-10 (Salmon et al., SC'11) at counters {block, walker, uid low, uid high | domain << 24}."""
    m32 = np.uint64(0xFFFFFFFF)
    c = [block.astype(np.uint64), walker.astype(np.uint64), uid & m32, (uid >> np.uint64(32)) & np.uint64(0xFFFFFF) | np.uint64(domain << 24)]
    k0, k1 = key & 0xFFFFFFFF, key >> 32
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & m32, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & m32]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return np.stack(c)


def _csr(n, src, dst, w):
    """Rows in edge-list order: an edge enters its source's row, then its target's."""
    rows, cols = np.stack([src, dst], 1).ravel().astype(np.int64), np.stack([dst, src], 1).ravel().astype(np.int64)
    order = np.argsort(rows, kind="stable")
    ptr = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(rows, minlength=n), out=ptr[1:])
    return ptr, cols[order], np.repeat(w, 2)[order]


def _walk(csr, src, dst, we, uid, case, seed, domain, threshold):
    """1/R of each edge's winning walk, 0 where no walk arrives.  The moves and the stops are those of the walks in
    32 bits (they are decisions); the path resistance is summed and inverted in 64."""
    ptr, col, w = csr
    r32, r64 = (np.float32(1.0) / w).astype(np.float32), 1.0 / w.astype(np.float64)
    W = case["walkers"]
    e = np.repeat(np.arange(len(src)), W)
    k = np.tile(np.arange(W), len(src))
    cur, prev = src[e].astype(np.int64), np.full(len(e), -1, np.int64)
    R, R64 = np.zeros(len(e), np.float32), np.zeros(len(e))
    won = []
    for step in range(1, case["steps"] + 1):
        if step >= case["steps"] and step > 1 or not len(e):
            break
        if (step - 1) % 4 == 0:
            draws = _philox(np.full(len(e), (step - 1) // 4), k, uid[e], domain, seed)
        deg = ptr[cur + 1] - ptr[cur]
        ok = deg >= (1 if step == 1 else 2)
        e, k, cur, prev, R, R64, deg, draws = e[ok], k[ok], cur[ok], prev[ok], R[ok], R64[ok], deg[ok], draws[:, ok]
        at = ptr[cur] + draws[(step - 1) % 4].astype(np.int64) % (deg if step == 1 else deg - 1)
        if step > 1:
            at = np.where(col[at] == prev, ptr[cur + 1] - 1, at)
        R, R64, nxt = (R + r32[at]).astype(np.float32), R64 + r64[at], col[at]
        alive = np.ones(len(e), bool) if step == 1 or threshold is None else ~((R * we[e]).astype(np.float32) >= threshold)
        hit = alive & (nxt == dst[e])
        won.append((e[hit], (np.float32(1.0) / R[hit]).astype(np.float32), k[hit], R64[hit]))
        alive &= ~hit
        e, k, prev, cur, R, R64, draws = e[alive], k[alive], cur[alive], nxt[alive], R[alive], R64[alive], draws[:, alive]
    out = np.zeros(len(src))
    if won:
        e, c, k, r = (np.concatenate(a) for a in zip(*won))
        order = np.lexsort((k, -c.astype(np.float64), e))
        first, at = np.unique(e[order], return_index=True)
        out[first] = 1.0 / r[order][at]
    return out


def _delete(csr, dels):
    """The rows after a batch of deletions, each moving its row's last slot into the hole."""
    ptr, col, w = csr
    rows = {int(v): [list(col[ptr[v]:ptr[v + 1]]), list(w[ptr[v]:ptr[v + 1]])] for v in np.unique(np.concatenate(dels))}
    for a, b in zip(*dels):
        for x, y in ((int(a), int(b)), (int(b), int(a))):
            cs, ws = rows[x]
            if y in cs:
                j = cs.index(y)
                cs[j], ws[j] = cs[-1], ws[-1]
                cs.pop()
                ws.pop()
    deg = np.diff(ptr)
    keep = np.ones(len(col), bool)
    col, w = col.copy(), w.copy()
    for v, (cs, ws) in rows.items():
        col[ptr[v]:ptr[v] + len(cs)], w[ptr[v]:ptr[v] + len(cs)] = cs, ws
        keep[ptr[v] + len(cs):ptr[v + 1]] = False
        deg[v] = len(cs)
    return np.concatenate([[0], np.cumsum(deg)]), col[keep], w[keep]


def exact(case, seed):
    """The conductances in 64 bits, by plain numpy walks; whole numbers have no other value in 64 bits.  None where
    that takes long or needs the recovered paths of earlier batches (deletions in several batches)."""
    if case["kind"] != "update" or case["transition"] != UNIFORM or case["walkers"] * (case["ins"] + case["dels"]) > 3_000_000:
        return None
    batch = case["batch"]
    if case["dels"] and (batch if batch else -(-case["dels"] // 10)) < case["dels"]:
        return None
    seed = 1000 * int(seed) + 17
    x = _lattice(case, seed)
    hs, hd, hw = (np.asarray(a) for a in x["h"])
    out = {}
    src, dst, w = x["ins"]
    if len(src):
        B = batch if batch else -(-len(src) // 10)
        cond = np.zeros(len(src))
        for b in range(0, len(src), B):
            sl = slice(b, min(b + B, len(src)))
            uid = np.arange(sl.start, sl.stop, dtype=np.uint64)
            cond[sl] = _walk(_csr(x["n"], hs, hd, hw), src[sl], dst[sl], w[sl], uid, case, seed, 0, np.float32(case["threshold"]))
            new = cond[sl] == 0
            hs, hd, hw = (np.concatenate([a, v[sl][new]]) for a, v in ((hs, src), (hd, dst), (hw, w)))
        out |= {"found_at": None, "conductance": cond, "accepted": None}
    if len(x["dels"][0]):
        gs, gd, gw = (np.concatenate([a, v]) for a, v in zip(x["g"], x["ins"]))
        a, b = np.minimum(*x["dels"]), np.maximum(*x["dels"])
        code = lambda u, v: np.minimum(u, v).astype(np.int64) * x["n"] + np.maximum(u, v)  # noqa: E731
        in_h = np.isin(code(a, b), code(hs, hd))
        cond = np.zeros(len(a))
        cond[in_h] = _walk(_delete(_csr(x["n"], gs, gd, gw), (a, b)), a[in_h], b[in_h], None,
                           np.flatnonzero(in_h).astype(np.uint64), case, seed, 1, None)
        out |= {"status": None, "del_conductance": cond, "rec_src": None, "rec_dst": None, "rec_kind": None,
                "n_rec": None}
    return out
