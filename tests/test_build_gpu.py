"""Parity of the CUDA SVG construction with the reference (GPU).

Bit-exact: neighbour sets, edge lengths and path-end fields of every row
must equal the reference's (golden fixtures) or the oracle's (the C
restatement pinned to the reference) on the same inputs.
"""
import os
import tempfile

import numpy as np
import pytest

from oracle.refbind import CpuOracle
from svg_b200 import MODE_BATCHED, MODE_PLAIN, SVG, Mesh, meshgen
from svg_b200.build_ext import build as build_lib
from tests.helpers import compare_rows, golden_params, load_golden, rows_from_padded, svg_file_bytes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib():
    build_lib()


def gpu_build(pos, faces, K, mode=MODE_BATCHED, **kw):
    m = Mesh.from_arrays(pos, faces)
    s = SVG()
    s.AssignMesh(m)
    s.SetParameters(K, kw.pop("split_coef", 10), kw.pop("vert_coef", 2))
    st = s.ConstructSVG(mode=mode, **kw)
    off, nodes = s.CopySVGToHost()
    return off, nodes, st, s, m


@pytest.mark.parametrize("mode", [MODE_BATCHED, MODE_PLAIN])
@pytest.mark.parametrize("name,K", golden_params())
def test_build_matches_reference_golden(name, K, mode):
    """Rows bit-exact against the reference.  Where the reference's fixed
    vertex/split hash tables (K*2, K*10 slots) overflow into their shared sink
    slot, the reference's search is no longer an ICH; such sources must be
    flagged (bit 2) and are excluded, their counters too."""
    g = load_golden(name)
    off, nodes, st, s, _ = gpu_build(g["pos"], g["faces"], K, mode)
    _, _, flags = s.source_stats()
    goff, gnodes = rows_from_padded(g[f"K{K}_tails"], g[f"K{K}_nodes"])
    ok_rows = [r for r in range(len(off) - 1) if not (flags[r] & 2)]
    assert compare_rows(off, nodes, goff, gnodes, rows=ok_rows) == []
    if st["ref_overflow_sources"] == 0:
        assert st["windows_generated"] == int(g[f"K{K}_stats"][:, 0].sum())
    assert st["watchdog_sources"] == 0


@pytest.mark.parametrize("n,blocks", [(1, 0), (2, 0), (4, 1), (5, 1), (9, 1), (127, 1), (128, 1), (129, 1), (300, 2),
                                      (1185, 0), (1500, 0)])
def test_sources_spread_over_warps_keep_their_rows(n, blocks):
    """Fewer sources than lanes run a few to a warp (1, 2, 3, ... 32 active
    lanes, one source more than the lanes, whole warps with none): the rows of
    the plain form, whose sources run one per thread."""
    pos, faces = meshgen.config_mesh(0, 0.25)
    out = []
    for mode, kw in ((MODE_PLAIN, {}), (MODE_BATCHED, dict(blocks=blocks))):
        off, nodes, st, _, _ = gpu_build(pos, faces, 40, mode, source_begin=100, source_end=100 + n, **kw)
        assert st["sources"] == n
        out.append((off, nodes))
    assert compare_rows(*out[0], *out[1]) == []


@pytest.mark.parametrize("n,blocks", [(128, 1), (129, 1), (255, 1), (257, 1), (700, 2), (1600, 3)])
def test_strided_work_order_keeps_the_rows(n, blocks):
    """More sources than a launch's lanes (128 per block), or just as many: the
    first wave strided over the warps in vertex order, then in the order of the
    first build's costs; every source is built once, with the plain form's rows."""
    pos, faces = meshgen.config_mesh(1, 0.2)
    m = Mesh.from_arrays(pos, faces)
    s = SVG()
    s.AssignMesh(m)
    s.SetParameters(30)
    s.ConstructSVG(mode=MODE_PLAIN, source_begin=7, source_end=7 + n)
    want = s.CopySVGToHost()
    for _ in range(3):
        st = s.ConstructSVG(blocks=blocks, heavy_first=1, source_begin=7, source_end=7 + n)
        assert st["sources"] == n
        assert compare_rows(*s.CopySVGToHost(), *want) == []


def coop_build(pos, faces, K, coop_warps=8, coop_sources=None, **kw):
    """Batched build whose work order comes from a first build's per-source
    costs, with the heaviest `coop_sources` (default: every source) run by
    whole warps (the cooperative form)."""
    m = Mesh.from_arrays(pos, faces)
    s = SVG()
    s.AssignMesh(m)
    s.SetParameters(K, kw.pop("split_coef", 10), kw.pop("vert_coef", 2))
    s.ConstructSVG(heavy_first=0, **kw)   # records the per-source costs on the mesh
    n = len(pos) if coop_sources is None else coop_sources
    st = s.ConstructSVG(heavy_first=1, coop_sources=n, coop_warps=coop_warps, **kw)
    off, nodes = s.CopySVGToHost()
    return off, nodes, st, s, m


@pytest.mark.parametrize("name,K", golden_params())
def test_cooperative_form_matches_reference_golden(name, K):
    """Every source run by a whole warp: the same rows as the reference."""
    g = load_golden(name)
    off, nodes, st, s, _ = coop_build(g["pos"], g["faces"], K)
    assert st["coop_sources"] == len(g["pos"])
    _, _, flags = s.source_stats()
    goff, gnodes = rows_from_padded(g[f"K{K}_tails"], g[f"K{K}_nodes"])
    ok_rows = [r for r in range(len(off) - 1) if not (flags[r] & 2)]
    assert compare_rows(off, nodes, goff, gnodes, rows=ok_rows) == []
    if st["ref_overflow_sources"] == 0:
        assert st["windows_generated"] == int(g[f"K{K}_stats"][:, 0].sum())


@pytest.mark.parametrize("cfg,K,n", [(1, 500, 1200), (0, 100, 1500)])
def test_cooperative_form_matches_oracle_on_benchmark_mesh_samples(cfg, K, n):
    """The heaviest sources of a leading source range run cooperatively (with
    the 1023-entry queue cap binding at K=500), the rest one per lane."""
    pos, faces = meshgen.config_mesh(cfg)
    off, nodes, st, _, _ = coop_build(pos, faces, K, coop_warps=32, coop_sources=n // 3,
                                      source_begin=0, source_end=n)
    assert st["coop_sources"] == n // 3
    (ooff, onodes), rows = _oracle_rows(pos, faces, K, np.arange(0, n, dtype=np.int32))
    assert compare_rows(off[:n + 1], nodes[:off[n]], ooff, onodes) == []
    assert st["windows_generated"] == int(rows.stats[:, 0].sum())


@pytest.mark.parametrize("cap,factor,coop", [(1472, 3, 100), (1473, 3, 100), (2047, 3, 100),
                                             (12928, 26, 100), (12929, 26, 0)])
def test_cooperative_heaps_of_every_size_are_built(cap, factor, coop):
    """Cooperative heaps just within and beyond what a block gets unasked beside
    the lanes' state (48 KB in all), the largest that can be asked for (227 KB in
    all), and one entry more, which leaves the sources to the lanes: the rows of a
    build without cooperative warps."""
    pos, faces = meshgen.config_mesh(1, 0.3)
    kw = dict(win_queue_cap=cap, heap_factor=factor, source_begin=0, source_end=300)
    off, nodes, st, _, _ = coop_build(pos, faces, 500, coop_warps=8, coop_sources=100, **kw)
    assert st["coop_sources"] == coop
    want = gpu_build(pos, faces, 500, **kw)
    assert compare_rows(off, nodes, want[0], want[1]) == []


def test_automatic_cooperative_share_keeps_the_graph():
    """The automatic choice (heaviest sources above a lane's average share)
    gives the same CSR as a build with no cooperative warps."""
    pos, faces = meshgen.config_mesh(1, 0.3)
    outs, counts = [], []
    for coop in (0, -1):
        m = Mesh.from_arrays(pos, faces)
        g = SVG()
        g.AssignMesh(m)
        g.SetParameters(300)
        g.ConstructSVG(heavy_first=0)
        st = g.ConstructSVG(heavy_first=1, coop_sources=coop)
        counts.append(st["coop_sources"])
        outs.append(g.csr())
    assert counts[0] == 0
    for x, y in zip(outs[0], outs[1]):
        assert np.array_equal(x, y)


def test_tail_adoption_keeps_the_graph():
    """Warps that adopt their last running lane's source once the queue is
    drained (the default) build the same CSR as warps that do not, and as
    the oracle on a sample of rows."""
    pos, faces = meshgen.config_mesh(1, 0.3)
    outs = []
    for tail in (0, 1):
        m = Mesh.from_arrays(pos, faces)
        g = SVG()
        g.AssignMesh(m)
        g.SetParameters(300)
        g.ConstructSVG(coop_tail=tail, heavy_first=0)
        outs.append(g.CopySVGToHost())
    assert compare_rows(outs[0][0], outs[0][1], outs[1][0], outs[1][1]) == []
    src = np.arange(0, len(pos), 37, dtype=np.int32)
    (ooff, onodes), _ = _oracle_rows(pos, faces, 300, src)
    off, nodes = outs[1]
    got_off = np.concatenate([[0], np.cumsum(np.diff(off)[src])])
    got = np.concatenate([nodes[off[v]:off[v + 1]] for v in src])
    assert compare_rows(got_off, got, ooff, onodes) == []


def test_build_replayed_from_a_captured_cuda_graph_is_identical():
    """opts.graph: the first build captures its device work as a CUDA graph
    kept with the mesh, later builds with the same options replay it; every
    result equals an ordinary build's rows (path ends included), also after
    another mesh's build has re-laid the lane scratch, and an option change
    builds the ordinary way."""
    pos, faces = meshgen.config_mesh(1, 0.3)
    ref_off, ref_nodes, _, _, _ = gpu_build(pos, faces, 200)
    m = Mesh.from_arrays(pos, faces)
    g = SVG()
    g.AssignMesh(m)
    g.SetParameters(200)
    replays = []
    for i in range(3):
        st = g.ConstructSVG(graph=1)
        replays.append(st["graph_replayed"])
        off, nodes = g.CopySVGToHost()
        assert compare_rows(off, nodes, ref_off, ref_nodes) == [], i
        if i == 1:  # another mesh and K re-lay the shared lane scratch
            other = SVG()
            other.AssignMesh(Mesh.from_arrays(*meshgen.torus(1.0, 0.35, 30, 20, 0.02, seed=5)))
            other.SetParameters(40)
            other.ConstructSVG()
    assert replays[0] == 0 and replays[1] == 1
    st = g.ConstructSVG(graph=1, vote_wait=4)  # other options: no replay
    assert st["graph_replayed"] == 0
    off, nodes = g.CopySVGToHost()
    assert compare_rows(off, nodes, ref_off, ref_nodes) == []


def test_autotuned_schedule_keeps_the_graph():
    """The tuner's candidates and its choice change the schedule only: the
    tuned build equals a default build bit for bit (the tuner itself also
    checks every candidate's CSR checksum against the first)."""
    pos, faces = meshgen.config_mesh(1, 0.25)
    m = Mesh.from_arrays(pos, faces)
    g = SVG()
    g.AssignMesh(m)
    g.SetParameters(200)
    g.ConstructSVG(heavy_first=0)
    ref = g.csr()
    best, ms = g.autotune(max_trials=12)
    assert best["autotune"] == 1 and ms > 0
    g.ConstructSVG(autotune=1)
    got = g.csr()
    for x, y in zip(ref, got):
        assert np.array_equal(x, y)


def test_reference_table_overflow_is_flagged():
    """monkey, K=6: the centre reaches 13 vertices, the reference's vertex
    table holds 2K = 12 keys."""
    g = load_golden("monkey")
    _, _, st, s, _ = gpu_build(g["pos"], g["faces"], 6)
    _, _, flags = s.source_stats()
    assert flags[0] & 2
    assert st["ref_overflow_sources"] >= 1


def _oracle_rows(pos, faces, K, src, **kw):
    rows = CpuOracle().mesh(pos, faces).build(K, src, threads=0, **kw)
    return rows_from_padded(rows.tails, rows.nodes), rows


@pytest.mark.parametrize("cfg,K,ranges", [
    (0, 100, [(0, 768), (15000, 15512)]),
    (1, 500, [(0, 300), (36300, 36556)]),
    (1, 100, [(72500, 72900)]),
])
def test_build_matches_oracle_on_benchmark_mesh_samples(cfg, K, ranges):
    pos, faces = meshgen.config_mesh(cfg)
    for a, b in ranges:
        off, nodes, st, _, m = gpu_build(pos, faces, K, source_begin=a, source_end=b)
        src = np.arange(a, b, dtype=np.int32)
        (ooff, onodes), rows = _oracle_rows(pos, faces, K, src)
        sub = off[a:b + 1] - off[a]
        got = nodes[off[a]:off[b]]
        assert compare_rows(sub, got, ooff, onodes) == []
        assert st["windows_generated"] == int(rows.stats[:, 0].sum())
        assert off[b] - off[a] == off[-1]  # rows outside the range are empty


def test_queue_capacity_drops_like_the_reference():
    pos, faces = meshgen.torus(1.0, 0.35, 24, 16, 0.02, seed=3)
    for mode in (MODE_BATCHED, MODE_PLAIN):
        off, nodes, st, _, _ = gpu_build(pos, faces, 30, mode, win_queue_cap=12, pseudo_queue_cap=5)
        (ooff, onodes), rows = _oracle_rows(pos, faces, 30, None, win_cap=12, pseudo_cap=5)
        assert compare_rows(off, nodes, ooff, onodes) == []
        assert st["queue_drop_sources"] > 0


def test_plain_and_batched_builds_are_identical():
    pos, faces = meshgen.height_field(40, seed=7)
    a = gpu_build(pos, faces, 60, MODE_BATCHED)
    b = gpu_build(pos, faces, 60, MODE_PLAIN)
    assert compare_rows(a[0], a[1], b[0], b[1]) == []
    assert a[2]["windows"] == b[2]["windows"]


def test_csr_without_paths_matches():
    pos, faces = meshgen.torus(1.0, 0.35, 30, 20, 0.02, seed=5)
    off, nodes, _, s, _ = gpu_build(pos, faces, 40, with_paths=False)
    coff, adj, dist = s.csr()
    (ooff, onodes), _ = _oracle_rows(pos, faces, 40, None)
    assert np.array_equal(coff, ooff)
    assert np.array_equal(adj, onodes["adj"])
    assert np.array_equal(dist, onodes["dist"])


def test_save_file_is_byte_identical_to_reference_format():
    g = load_golden("monkey")
    K = 20
    _, _, _, s, m = gpu_build(g["pos"], g["faces"], K)
    goff, gnodes = rows_from_padded(g[f"K{K}_tails"], g[f"K{K}_nodes"])
    with tempfile.TemporaryDirectory() as td:
        p = os.path.join(td, "m.svg")
        s.SaveSVGToFile(p)
        data = open(p, "rb").read()
        gn = gnodes.copy()
        gn["pad"] = 0
        assert data == svg_file_bytes(goff, gn)
        s2 = SVG()
        s2.AssignMesh(m)
        s2.SetParameters(K)
        s2.LoadSVGFromFile(p)
        off2, n2 = s2.CopySVGToHost()
        assert compare_rows(off2, n2, goff, gnodes) == []


def test_per_source_statistics():
    pos, faces = meshgen.torus(1.0, 0.35, 30, 20, 0.02, seed=5)
    _, _, st, s, _ = gpu_build(pos, faces, 40)
    w, q, f = s.source_stats()
    assert w.sum() == st["windows"]
    assert q.max() == st["max_win_queue"]
    assert (f == 0).all()


def test_bad_arguments_are_reported():
    from svg_b200 import SvgError
    pos, faces = meshgen.torus(1.0, 0.35, 8, 6, 0.02, seed=5)
    with pytest.raises(SvgError):
        gpu_build(pos, faces, 0)
    with pytest.raises(SvgError):
        gpu_build(pos, faces, 10, source_begin=10, source_end=5)


def test_work_order_does_not_change_the_graph():
    """Which lane builds which source, and when, is a scheduling choice: vertex
    order, heaviest-first from the previous build, and the K/10 probe order give
    the same CSR bit for bit."""
    import svg_b200
    from svg_b200 import SVG, Mesh
    pos, faces = meshgen.config_mesh(1, 0.3)
    outs = []
    for hf, warm in ((0, False), (1, True), (2, False)):
        m = Mesh.from_arrays(pos, faces)
        g = SVG()
        g.AssignMesh(m)
        g.SetParameters(200)
        if warm:
            g.ConstructSVG(heavy_first=0)   # leaves per-source costs on the mesh
        g.ConstructSVG(heavy_first=hf)
        outs.append(g.csr())
    for o in outs[1:]:
        for x, y in zip(outs[0], o):
            assert np.array_equal(x, y)
    mem = svg_b200.device_memory()
    assert mem["in_use"] > 0 and mem["peak"] >= mem["in_use"]


@pytest.mark.parametrize("K", [300, 1000, 1500])
def test_emission_of_short_and_long_candidate_lists(K):
    """Lists of up to 1,023 candidates are sorted as 32-bit keys, longer ones as
    64-bit keys (a dome: no saddle vertex, so every vertex reached is a
    candidate; sources near its middle): the plain form's rows."""
    k = 56
    rng = np.random.default_rng(3)
    y, x = np.mgrid[0:k, 0:k] + rng.uniform(-0.2, 0.2, (2, k, k))
    pos = np.stack([x, y, -0.004 * ((x - 28) ** 2 + (y - 28) ** 2)], -1).reshape(-1, 3)
    i = (np.arange(k - 1)[:, None] * k + np.arange(k - 1)).ravel()
    faces = np.concatenate([np.stack([i, i + 1, i + k], 1), np.stack([i + 1, i + k + 1, i + k], 1)]).astype(np.int32)
    out = [gpu_build(pos, faces, K, mode, source_begin=1500, source_end=1540)[:2] for mode in (MODE_BATCHED, MODE_PLAIN)]
    assert np.diff(out[0][0]).max() == K
    assert compare_rows(*out[0], *out[1]) == []


@pytest.mark.parametrize("with_paths", [True, False])
def test_rows_reach_the_host_without_device_memory(with_paths):
    """With 8 MB of the device left (a piece of the rows takes 20), the nodes are
    assembled on the host: the same rows, padding included, and the same file."""
    import gc

    import torch

    import svg_b200
    pos, faces = meshgen.torus(1.0, 0.35, 130, 100, 0.02, seed=5)
    off, nodes, _, s, _ = gpu_build(pos, faces, 40, with_paths=with_paths)
    assert 40 * len(nodes) > 16 << 20
    with tempfile.TemporaryDirectory() as td:
        s.SaveSVGToFile(os.path.join(td, "a"))
        gc.collect()
        svg_b200.lib().svg_trim_device_cache()
        torch.cuda.empty_cache()
        hold = torch.empty(torch.cuda.mem_get_info()[0] - (8 << 20), dtype=torch.uint8, device="cuda")
        try:
            off2, nodes2 = s.CopySVGToHost()
            s.SaveSVGToFile(os.path.join(td, "b"))
        finally:
            del hold
            torch.cuda.empty_cache()
        a, b = (open(os.path.join(td, x), "rb").read() for x in "ab")
    assert np.array_equal(off, off2) and nodes.tobytes() == nodes2.tobytes() and a == b


@pytest.mark.parametrize("blocks", [1, 2, 5])
def test_a_small_launch_uses_every_lane(blocks):
    """At K = 300 launches of the whole GPU make their waves equal by using fewer
    lanes of each warp; one of few blocks with one source more than its lanes
    keeps them all (the same scratch), and its rows."""
    pos, faces = meshgen.config_mesh(1, 0.2)
    lanes, scratch, rows = 128 * blocks, [], []
    for n in (lanes, lanes + 1):
        off, nodes, st, _, _ = gpu_build(pos, faces, 300, blocks=blocks, heavy_first=0, source_begin=0, source_end=n)
        scratch.append(st["scratch_bytes"])
        rows.append((off, nodes))
    assert scratch[0] == scratch[1]
    want = gpu_build(pos, faces, 300, source_begin=0, source_end=lanes + 1)
    assert compare_rows(*rows[1], *want[:2]) == []


def test_automatic_cooperative_share_counts_two_blocks_per_sm():
    """The sources that cost more than a lane's average share of the build are
    counted with the lanes of two blocks per SM, also where three run, and their
    rows stay."""
    import torch
    pos, faces = meshgen.config_mesh(1)
    m = Mesh.from_arrays(pos, faces)
    s = SVG()
    s.AssignMesh(m)
    s.SetParameters(50)
    s.ConstructSVG(heavy_first=0)
    want = s.csr()
    cost = s.source_stats()[0].astype(np.int64)
    st = s.ConstructSVG(heavy_first=1, coop_sources=-1)
    lanes = 2 * torch.cuda.get_device_properties(0).multi_processor_count * 128
    assert st["coop_sources"] == min((cost >= cost.sum() / lanes).sum(), lanes // 64)
    for x, y in zip(want, s.csr()):
        assert np.array_equal(x, y)


_NEARLY_FULL = """
import sys
import numpy as np, torch
from svg_b200 import SVG, Mesh, meshgen
pos, faces = meshgen.torus(1.0, 0.35, 1250, 800, 0.0, seed=1)
m = Mesh.from_arrays(pos, faces)
m.copyToGPU()
s = SVG()
s.AssignMesh(m)
s.SetParameters(10)
torch.empty(1, device="cuda")
hold = torch.empty(torch.cuda.mem_get_info()[0] - (3640 << 20), dtype=torch.uint8, device="cuda")
st = s.ConstructSVG()
got = s.csr()
print("scratch", st["scratch_bytes"])
del hold
torch.cuda.empty_cache()
want_st = s.ConstructSVG(blocks=2 * torch.cuda.get_device_properties(0).multi_processor_count)
assert st["scratch_bytes"] == want_st["scratch_bytes"]
assert all(np.array_equal(x, y) for x, y in zip(got, s.csr()))
"""


def test_a_build_without_room_for_three_blocks_per_sm_runs_two():
    """1 M sources at K = 10 with 3.6 GB of the device left: the scratch of three
    blocks per SM (1.8 GB, half of that) leaves no room for the candidates and
    rows, that of two does, as when two were all there were.  In a process of its
    own: scratch that an earlier build left would count."""
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _NEARLY_FULL], cwd=root, env=dict(os.environ, PYTHONPATH=root),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def test_launches_are_counted():
    """Work order (one kernel, three by cost, none for the host's), search, offsets
    scan, emission, path ends and flag tallies; plain: rows packed instead of
    emitted; replayed: no order."""
    pos, faces = meshgen.torus(1.0, 0.35, 30, 20, 0.02, seed=5)
    m = Mesh.from_arrays(pos, faces)
    s = SVG()
    s.AssignMesh(m)
    s.SetParameters(20)
    assert s.ConstructSVG()["launches"] == 6
    assert s.ConstructSVG(with_paths=False)["launches"] == 5
    assert s.ConstructSVG(mode=MODE_PLAIN)["launches"] == 5
    one = dict(blocks=1, threads_per_block=32, heavy_first=1)   # more sources than lanes
    uneven = dict(one, source_begin=0, source_end=60)           # fewer than 3.5 waves: by cost
    s.ConstructSVG(**uneven)
    assert s.ConstructSVG(**uneven)["launches"] == 8
    assert s.ConstructSVG(**uneven, coop_sources=2)["launches"] == 5
    s.ConstructSVG(graph=1)
    st = s.ConstructSVG(graph=1)
    assert st["graph_replayed"] == 1 and st["launches"] == 5


def test_three_blocks_of_the_build_kernel_run_per_sm():
    """A build of many sources launches three blocks per SM (its registers just
    allow it): the scratch of as many blocks asked for."""
    import torch
    pos, faces = meshgen.torus(1.0, 0.35, 300, 200, 0.02, seed=5)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    a = gpu_build(pos, faces, 10, heavy_first=0)[2]["scratch_bytes"]
    assert a == gpu_build(pos, faces, 10, heavy_first=0, blocks=3 * sms)[2]["scratch_bytes"]
