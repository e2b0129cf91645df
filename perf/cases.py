"""Performance cases of the Saddle Vertex Graph engine: what its users have it do.

A program builds the graph of a mesh (on the device, or down to the host's
reference-layout rows), then asks it single-pair (SSSD) and whole-graph
multi-source (MSAD) distances: one at a time, in batches, with path parents,
or through the serving loop.  Meshes are this package's seeded generators at
the sizes of its benchmark configurations (30K torus at K=100, 72.9K height
field at K=500, 750K noisy torus at K=100), of its mixed-serving pool
(5K to 300K vertices, K of 50 and 200) and of its small test meshes.
"""
from __future__ import annotations

import ctypes as C
import heapq
import math
import os
import tempfile

import numpy as np
import torch

from svg_b200 import NODE_DTYPE, SVG, Mesh, Server, lib, meshgen

MESHES = ("torus", "hfield", "noise")   # closed tube, open terrain, closed multi-octave tube
KS = (20, 50, 100, 200, 500)            # the K of the tests, the pool and the configurations
RING = 4                                # grid radius of a stored graph's rows: 80 neighbours


def listed():
    return [
        # an editor's small part: one build at interactive rate, bound by latency and launches
        dict(name="build_torus_600_K20", op="build", mesh="torus", nv=600, K=20, paths=True),
        # the serving pool's smallest mesh, rebuilt on demand
        dict(name="build_torus_5k_K50", op="build", mesh="torus", nv=5000, K=50, paths=True),
        # the 30K-vertex closed model of the first benchmark configuration
        dict(name="build_torus_30k_K100", op="build", mesh="torus", nv=30000, K=100, paths=True),
        # the headline benchmark: an uneven terrain with boundary at the largest K
        dict(name="build_hfield_73k_K500", op="build", mesh="hfield", nv=72900, K=500, paths=True),
        # the largest mesh, built for queries only (no path ends)
        dict(name="build_noise_750k_K100", op="build", mesh="noise", nv=750000, K=100, paths=False),
        # the reference driver's flow: construct, then copy the rows to the host
        dict(name="rows_hfield_12k_K200", op="rows", mesh="hfield", nv=12000, K=200, paths=True),
        # an interactive pick on a graph loaded from its file: one pair a call
        dict(name="sssd_1_stored_30k", op="sssd", mesh="torus", nv=30000, K=100, stored=True, n=1),
        # a batch job of point pairs on the largest graph
        dict(name="sssd_2048_noise_750k", op="sssd", mesh="noise", nv=750000, K=100, stored=False, n=2048),
        # one distance field on the largest graph
        dict(name="msad_1_noise_750k", op="msad", mesh="noise", nv=750000, K=100, stored=False, n=1, srcs=100),
        # a batch of distance fields (Voronoi-like labels) on a terrain
        dict(name="msad_32_hfield_73k", op="msad", mesh="hfield", nv=72900, K=200, stored=False, n=32, srcs=30),
        # distance fields with parents, for tracing paths, on a graph loaded from its file
        dict(name="msad_paths_4_stored_30k", op="msad_paths", mesh="torus", nv=30000, K=100, stored=True, n=4, srcs=5),
        # the serving loop: a burst of mixed requests on a resident graph
        dict(name="serve_200_torus_30k", op="serve", mesh="torus", nv=30000, K=100, stored=False, n=200),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: any operation, sizes log-uniform over the listed range,
    no dearer than the listed case of its kind."""
    op = rng.choice(("build", "build", "build", "build", "rows", "sssd", "sssd", "msad", "msad", "msad_paths", "serve"))
    mesh = rng.choice(MESHES)
    if op == "build":
        K = rng.choice(KS)
        nv = _log_int(rng, 200, min(750000, 0.9 * _windows(72900, 500) / _windows(1, K)))
        return dict(op=op, mesh=mesh, nv=nv, K=K, paths=rng.random() < 0.6)
    K = rng.choice((50, 100, 200))
    if op == "rows":
        return dict(op=op, mesh=mesh, nv=_log_int(rng, 200, 2400000 // K), K=K, paths=True)
    stored = rng.random() < 0.3
    nv = _log_int(rng, 500, 50000 if stored else 300000)
    K = 100 if stored else K
    mesh = "torus" if stored else mesh
    if op == "sssd":
        return dict(op=op, mesh=mesh, nv=nv, K=K, stored=stored, n=_log_int(rng, 1, 1000))
    if op == "serve":
        return dict(op=op, mesh=mesh, nv=min(nv, 60000), K=K, stored=stored, n=_log_int(rng, 10, 200))
    n = _log_int(rng, 1, max(1, min(32, 2400000 // nv)))
    return dict(op=op, mesh=mesh, nv=nv, K=K, stored=stored, n=n, srcs=_log_int(rng, 1, min(1000, nv // 4)))


# ------------------------------------------------------------------ inputs

def _grid(mesh, nv):
    """Grid (rows, columns) of a mesh of about nv vertices."""
    if mesh == "hfield":
        n = max(8, int(round(math.sqrt(nv))))
        return n, n
    cols = max(8, int(round(math.sqrt(nv * 0.75))))
    return max(8, int(round(nv / cols))), cols


def _arrays(mesh, nv, seed):
    nu, n = _grid(mesh, nv)
    if mesh == "hfield":
        return meshgen.height_field(n, seed=seed)
    if mesh == "torus":
        return meshgen.torus(1.0, 0.35, nu, n, 0.02, seed=seed)
    return meshgen.torus_value_noise(1.0, 0.4, nu, n, seed=seed)


def _stored_graph(pos, nu, n):
    """Rows of a stored graph of a torus grid: every vertex joined to those up
    to RING grid steps away, by the straight length (CSR, ascending rows)."""
    V = nu * n
    di, dj = np.meshgrid(np.arange(-RING, RING + 1), np.arange(-RING, RING + 1), indexing="ij")
    keep = (di != 0) | (dj != 0)
    di, dj = di[keep], dj[keep]
    i, j = np.divmod(np.arange(V), n)
    adj = ((i[:, None] + di[None]) % nu) * n + (j[:, None] + dj[None]) % n
    adj = np.sort(adj, axis=1)
    d = pos[adj] - pos[:, None]
    return adj.astype(np.int32), np.sqrt((d * d).sum(-1))


def _save_rows(path, adj, dist):
    """The reference's graph file: per vertex an int32 degree, then its nodes."""
    row = np.dtype([("deg", np.int32), ("nodes", NODE_DTYPE, (adj.shape[1],))])
    out = np.zeros(len(adj), row)
    out["deg"] = adj.shape[1]
    out["nodes"]["adj"] = adj
    out["nodes"]["dist"] = dist
    out["nodes"]["src_edge"] = out["nodes"]["dst_edge"] = 0xFFFFFFFF
    out.tofile(path)


def _queries(case, V, rng):
    """The query part of a state: pairs, or weighted source sets."""
    if case["op"] == "sssd":
        return dict(s=rng.integers(0, V, case["n"]).astype(np.int32), t=rng.integers(0, V, case["n"]).astype(np.int32))
    if case["op"] == "serve":
        reqs = []
        for i in range(case["n"]):
            if i % 10 not in (2, 5, 8):
                reqs.append((int(rng.integers(0, V)), int(rng.integers(0, V))))
            else:
                k = min(V // 4, int(round(math.exp(rng.uniform(0.0, math.log(1000.0))))))
                reqs.append(rng.choice(V, k, replace=False).astype(np.int32))
        return dict(reqs=reqs)
    sets = [rng.choice(V, case["srcs"], replace=False).astype(np.int32) for _ in range(case["n"])]
    return dict(sets=sets, weights=[rng.uniform(0.0, 0.05, case["srcs"]) for _ in sets])


def prepare(case, seed):
    pos, faces = _arrays(case["mesh"], case["nv"], seed)
    m = Mesh.from_arrays(pos, faces)
    m.copyToGPU()
    svg = SVG()
    svg.AssignMesh(m)
    svg.SetParameters(case["K"])
    st = dict(op=case["op"], svg=svg, paths=case.get("paths", False))
    room = m.vertNum * case["K"]         # a row has at most K edges
    if case["op"] == "build":
        st["csr"] = [torch.zeros(k, dtype=t, device="cuda") for k, t in
                     ((m.vertNum + 1, torch.int64), (room, torch.int32), (room, torch.float64))]
        return st
    if case["op"] == "rows":
        st["tails"], st["nodes"] = np.zeros(m.vertNum, np.int32), np.zeros(room, NODE_DTYPE)
        return st
    if case["stored"]:
        fd, path = tempfile.mkstemp(suffix=".svg")
        os.close(fd)
        try:
            _save_rows(path, *_stored_graph(pos, *_grid(case["mesh"], case["nv"])))
            svg.LoadSVGFromFile(path)
        finally:
            os.remove(path)
    else:
        svg.ConstructSVG(with_paths=False)
    st.update(_queries(case, m.vertNum, np.random.default_rng(seed)))
    if case["op"] == "serve":
        st["server"] = Server(staging_in_bytes=1 << 20, staging_out_bytes=16 << 20)
        st["gid"] = st["server"].add_graph(svg)
        n_msad = sum(not isinstance(r, tuple) for r in st["reqs"])
        st["dist"] = np.zeros((n_msad, m.vertNum))
        st["src"] = np.zeros((n_msad, m.vertNum), np.int32)
    return st


# ------------------------------------------------------------------ passes

class _DeviceArray:
    """A device pointer as torch.as_tensor takes it (no copy)."""

    def __init__(self, ptr, n, typestr):
        self.__cuda_array_interface__ = dict(shape=(n,), typestr=typestr, data=(ptr, False), version=3)


def _ok(status):
    if status != 0:
        raise RuntimeError(lib().svg_last_error().decode())


def _copy_device_csr(svg, out):
    """The resident graph's CSR into the program's own tensors (room for full
    rows), which outlive the graph: the next build frees it."""
    p = [C.c_void_p() for _ in range(3)]
    _ok(lib().svg_graph_device_csr(svg._g, *[C.byref(x) for x in p]))
    nv, nnz, _ = svg.counts()
    for x, n, t, o in zip(p, (nv + 1, nnz, nnz), ("<i8", "<i4", "<f8"), out):
        o[:n].copy_(torch.as_tensor(_DeviceArray(x.value, n, t), device="cuda"))
    return out


def run(state):
    op, svg = state["op"], state["svg"]
    if op == "build":
        svg.ConstructSVG(with_paths=state["paths"])
        return _copy_device_csr(svg, state["csr"])
    if op == "rows":                     # into the program's own host rows
        svg.ConstructSVG(with_paths=True)
        tails, nodes = state["tails"], state["nodes"]
        _ok(lib().svg_graph_copy_nodes(svg._g, tails.ctypes.data_as(C.c_void_p), nodes.ctypes.data_as(C.c_void_p)))
        return [tails] + [nodes[f] for f in ("adj", "dist", "src_edge", "dst_edge", "src_x", "dst_x")]
    if op == "sssd":
        return svg.sssd_batch(state["s"], state["t"])
    if op == "msad":
        return svg.msad_batch(state["sets"], state["weights"])
    if op == "msad_paths":
        return svg.msad_paths(state["sets"], state["weights"])
    srv, gid, tickets, k = state["server"], state["gid"], [], 0
    for r in state["reqs"]:
        if isinstance(r, tuple):
            tickets.append(srv.submit_sssd(gid, *r))
        else:
            tickets.append(srv.submit_msad(gid, r, out=(state["dist"][k], state["src"][k])))
            k += 1
    got = []
    for t, r in zip(tickets, state["reqs"]):
        d = srv.wait(t)["dist"]
        srv.take(t)
        if isinstance(r, tuple):
            got.append(d)
    return [np.array(got), state["dist"], state["src"]]


# ------------------------------------------------------------------ bounds

def _windows(nv, K):
    """Windows a build propagates: about 5 K per source at K = 100, 17 K at 500."""
    return nv * K * (2.0 + 0.03 * K)


def work(case):
    nu, n = _grid(case["mesh"], case["nv"])
    V, K, op = nu * n, case["K"], case["op"]
    geometry = 24 * V + 24 * V           # positions, and two faces of 12 bytes a vertex
    edges = 0.8 * K * V
    if op in ("build", "rows"):
        per_edge = 40 if op == "rows" else (36 if case["paths"] else 12)
        return dict(bytes=geometry + per_edge * edges + 8 * V, flops=300.0 * _windows(V, K))
    if op == "sssd":                     # the edges a search meets on its way depend on the pair: about a tenth
        return dict(bytes=case["n"] * (0.1 * 12 * edges + 16), flops=case["n"] * 0.1 * 2 * edges)
    if op == "serve":
        return dict(bytes=case["n"] * (0.7 * 0.1 + 0.3) * 12 * edges + 0.3 * case["n"] * 12 * V,
                    flops=case["n"] * 0.37 * 2 * edges)
    per_vertex = 16 if op == "msad_paths" else 12
    return dict(bytes=case["n"] * (12 * edges + per_vertex * V), flops=case["n"] * 2 * edges)


def _dijkstra(adj, dist, srcs, weights, target=None):
    d = np.full(len(adj), np.inf)
    d[srcs] = weights
    heap = [(float(d[s]), int(s)) for s in set(srcs.tolist())]
    heapq.heapify(heap)
    while heap:
        du, u = heapq.heappop(heap)
        if du > d[u]:
            continue
        if u == target:
            break
        nd = du + dist[u]
        better = nd < d[adj[u]]
        for v, x in zip(adj[u][better].tolist(), nd[better].tolist()):
            d[v] = x
            heapq.heappush(heap, (x, v))
    return np.where(np.isfinite(d), d, np.finfo(np.float64).max)


def exact(case, seed):
    """Distances on stored graphs by Dijkstra (source labels and parents may
    name any of several equal ones: no value).  A graph built from a mesh has
    no short independent form."""
    op = case["op"]
    if op in ("build", "rows") or not case["stored"] or case["n"] * case["nv"] > 200000:
        return None
    pos, _ = _arrays(case["mesh"], case["nv"], seed)
    nu, n = _grid(case["mesh"], case["nv"])
    adj, dist = _stored_graph(pos, nu, n)
    q = _queries(case, nu * n, np.random.default_rng(seed))
    if op == "sssd":
        return np.array([_dijkstra(adj, dist, np.array([s]), np.zeros(1), int(t))[t] for s, t in zip(q["s"], q["t"])])
    if op == "serve":
        pairs = [r for r in q["reqs"] if isinstance(r, tuple)]
        sets = [r for r in q["reqs"] if not isinstance(r, tuple)]
        one = [_dijkstra(adj, dist, np.array([s]), np.zeros(1), t)[t] for s, t in pairs]
        return [np.array(one), np.array([_dijkstra(adj, dist, s, np.zeros(len(s))) for s in sets]).reshape(-1, nu * n), None]
    full = np.array([_dijkstra(adj, dist, s, w) for s, w in zip(q["sets"], q["weights"])])
    return [full, None] if op == "msad" else [full, None, None]
