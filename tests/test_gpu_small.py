"""The one-launch steps of small graphs, and the launch-per-step sweeps of
middle-sized ones, against the general kernels.

A probe limit that no table reaches sends the same calls through the general
path (one launch per step, compared with the CPU oracle by the parity tests),
so both paths of the library see the same inputs and must give the same bits.
"""
import contextlib

import numpy as np
import pytest

import pennsylvaniagpugraphclustering_b200 as pg
from oracle import mlp_oracle as M
from pennsylvaniagpugraphclustering_b200 import _lib
from pennsylvaniagpugraphclustering_b200 import move_filter as MF
from pennsylvaniagpugraphclustering_b200.graphgen import HostGraph

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def general_path(mem):
    _lib.check(_lib.lib().pggc_debug_set_probe_limit(mem.handle, 1 << 30))
    try:
        yield
    finally:
        _lib.check(_lib.lib().pggc_debug_set_probe_limit(mem.handle, 0))


def _graph(n, pairs, weights, seed):
    """Symmetric CSR of random pairs; weights: None, "int", "signed" or "float" (multiples of 2^-24)."""
    rng = np.random.default_rng(seed)
    u, v = pairs
    keep = u != v
    key = np.unique(np.concatenate([u[keep] * n + v[keep], v[keep] * n + u[keep]]))
    src, dst = key // n, key % n
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.int64)
    w = None
    if weights:
        lo, hi = np.minimum(src, dst), np.maximum(src, dst)
        _, inv = np.unique(lo * n + hi, return_inverse=True)
        k = int(inv.max()) + 1 if len(inv) else 1
        if weights == "float":
            w = (0.5 + rng.integers(0, 1 << 24, k) * 2.0 ** -24).astype(np.float32)[inv]
        else:
            w = rng.integers(-2 if weights == "signed" else 1, 9, k).astype(np.int32)[inv]
    return HostGraph(rowptr, dst.astype(np.int32), w)


def _planted(n, block, deg_in, deg_out, seed, hubs=0, hub_deg=0):
    """Pairs of a planted partition, `hubs` vertices with hub_deg more neighbours."""
    rng = np.random.default_rng(seed)
    u = rng.integers(0, n, int(n * deg_in / 2))
    v = np.minimum(u // block * block + rng.integers(0, block, len(u)), n - 1)
    a, b = rng.integers(0, n, (2, int(n * deg_out / 2)))
    h = np.repeat(np.arange(hubs) * 7 % n, hub_deg)
    t = rng.integers(0, n, len(h))
    return np.concatenate([u, a, h]).astype(np.int64), np.concatenate([v, b, t]).astype(np.int64)


# name: (vertices, block, deg_in, deg_out, hubs, hub degree)
FORMS = {
    "one_vertex": (1, 1, 0, 0, 0, 0),
    "no_edges": (40, 8, 0, 0, 0, 0),
    "warp_edge": (33, 8, 6, 1, 0, 0),
    "chunk_edge": (1025, 40, 8, 3, 0, 0),
    "classes_0_to_3": (2000, 50, 14, 4, 60, 60),
    "rows_128_warp_tables": (700, 350, 200, 40, 0, 0),       # labels fit a warp's share
    "rows_128_block_tables": (3000, 60, 10, 4, 40, 400),      # they do not
    "rows_4096": (30000, 60, 2, 1, 3, 5500),                  # several passes of the table
    "largest_move": (32768, 128, 2, 1.5, 0, 0),               # the most vertices, few edges
    "move_16k": (16000, 128, 2, 1, 0, 0),                     # close to the one-launch move's limit
    "largest": (32768, 128, 5, 2, 0, 0),                      # one launch for contraction and refinement
    "steps_40k": (40000, 100, 9, 3, 30, 400),                 # a launch per step
    "steps_hubs": (50000, 60, 6, 2, 3, 6000),
    "star_of_14000": (14001, 1, 0, 0, 1, 60000),              # a tree of thousands
}


def _host_graph(form, weights):
    n, block, din, dout, hubs, hdeg = FORMS[form]
    return _graph(n, _planted(n, max(block, 1), din, dout, 3, hubs, hdeg), weights, 5)


def _objective(weights):
    return pg.OBJ_MOD if weights is None else pg.OBJ_WMOD


def _wgraph(mem, hg, weights):
    return pg.weighted_graph(mem, hg.rowptr, hg.col, hg.w, objective=_objective(weights))


@pytest.mark.parametrize("weights", [None, "int", "signed", "float"])
@pytest.mark.parametrize("form", list(FORMS))
def test_local_move(mem, form, weights):
    hg = _host_graph(form, weights)
    g = _wgraph(mem, hg, weights)

    def moves():
        out = []
        rfd = pg.get_objective(mem, g, _objective(weights))
        part = np.arange(g.n, dtype=np.int32)
        for initial, sa, limit in ((True, True, -1), (False, True, 3), (False, False, -1)):
            st = pg.local_move(mem, g, part, rfd, initial, enable_simulated_annealing=sa, sweep_limit=limit)
            out.append((part.copy(), st["sweeps"], st["moves"], rfd.obj, rfd.uncut, rfd.label_count,
                        rfd.total_deg()))
        # from a partition that mixes the communities, constrained to halves
        mixed = (np.arange(g.n, dtype=np.int32) % max(1, min(g.n, 37))).astype(np.int32)
        con = (np.arange(2 * g.n + 64) % 2).astype(np.int32)
        vw = g.to_host()[3]
        td = np.zeros(int(mixed.max()) + 1, vw.dtype)
        np.add.at(td, mixed, vw)
        rfd.set_state(len(td), td, 0.0)
        st = pg.local_move(mem, g, mixed, rfd, False, constraint=con)
        out.append((mixed, con, st["moves"], rfd.obj, rfd.label_count))
        return out

    got = moves()
    with general_path(mem):
        want = moves()
    for a, b in zip(got, want):
        for x, y in zip(a, b):
            np.testing.assert_array_equal(x, y)  # NaN objectives (no edges) are equal


@pytest.mark.parametrize("weights", [None, "int", "float"])
@pytest.mark.parametrize("form", list(FORMS))
def test_strict_and_refinement(mem, form, weights):
    hg = _host_graph(form, weights)
    g = _wgraph(mem, hg, weights)

    def steps():
        out = []
        rfd = pg.get_objective(mem, g, _objective(weights))
        part = np.arange(g.n, dtype=np.int32)
        for sweeps in (1, -1, -1):  # after one sweep many candidates are left, at the end few or none
            pg.local_move(mem, g, part, rfd, sweeps == 1, sweep_limit=sweeps)
            vcmap, nc = pg.coarsen_leidenR(mem, g, part, rfd, 11 + sweeps, 5)
            out.append((vcmap, nc))
            st = pg.local_move_strict(mem, g, part, rfd, False)
            out.append((part.copy(), st["sweeps"], st["moves"], rfd.obj, rfd.label_count))
        con = (np.arange(2 * g.n + 64) % 2).astype(np.int32)
        st = pg.local_move_strict(mem, g, part, rfd, False, constraint=con)
        # one tree per star, up to the whole graph
        one = np.zeros(g.n, np.int32)
        rfd.set_state(1, np.array([rfd.total_deg().sum()]), 0.0)
        out.append((part, st["moves"], *pg.coarsen_leidenR(mem, g, one, rfd, 3, 4)))
        return out

    got = steps()
    with general_path(mem):
        want = steps()
    for a, b in zip(got, want):
        for x, y in zip(a, b):
            np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("weights", [None, "int", "signed", "float"])
@pytest.mark.parametrize("form,nc", [("one_vertex", 1), ("no_edges", 7), ("warp_edge", 33), ("chunk_edge", 1),
                                     ("chunk_edge", 1024), ("chunk_edge", 1025), ("classes_0_to_3", 31),
                                     ("rows_128_block_tables", 1500), ("rows_4096", 16385), ("rows_4096", 30000),
                                     ("largest", 1100), ("largest", 20000)])
def test_contraction(mem, form, nc, weights):
    hg = _host_graph(form, weights)
    g = _wgraph(mem, hg, weights)
    rng = np.random.default_rng(nc)
    # every id used, one large cluster and many small ones
    vcmap = np.concatenate([np.arange(nc), np.where(rng.random(g.n - nc) < 0.3, 0, rng.integers(0, nc, g.n - nc))])
    vcmap = rng.permutation(vcmap).astype(np.int32)
    got = pg.build_coarse_graph(mem, g, vcmap, nc)
    with general_path(mem):
        want = pg.build_coarse_graph(mem, g, vcmap, nc)
        # the next level's products come with the small path's graph
        o_want = pg.generate_orderings(mem, want)
    assert got.nnz == want.nnz
    for a, b in zip(got.to_host(), want.to_host()):
        assert np.array_equal(a, b)
    assert all(np.array_equal(a, b) for a, b in zip(pg.generate_orderings(mem, got), o_want))


@pytest.mark.parametrize("method", [pg.METHOD_LOUVAIN, pg.METHOD_LEIDEN, pg.METHOD_LEIDEN_PLUS])
@pytest.mark.parametrize("form,weights", [("chunk_edge", None), ("classes_0_to_3", "float"),
                                          ("rows_128_block_tables", "int"), ("largest_move", "float"), ("largest", "float"),
                                          ("move_16k", "int"),
                                          ("steps_40k", "float"), ("steps_hubs", "int")])
def test_runs(mem, form, weights, method):
    hg = _host_graph(form, weights)
    g = _wgraph(mem, hg, weights)

    def run():
        rfd = pg.get_objective(mem, g, _objective(weights))
        labels, st = pg.run_clustering(mem, g, rfd, method=method, ex_iters=0 if method == pg.METHOD_LOUVAIN else 1,
                                       seed=9)
        return labels, {k: v for k, v in st.items()}

    got = run()
    with general_path(mem):
        want = run()
    assert np.array_equal(got[0], want[0]) and got[1] == want[1]


@pytest.mark.parametrize("blocks", [15, 8, 7, 0])
@pytest.mark.parametrize("form", ["one_vertex", "classes_0_to_3", "rows_128_block_tables", "move_16k"])
def test_device_that_places_no_large_cluster(mem, form, blocks):
    """Clusters of 8 where 16 cannot be placed, the general path below: the same answers from every step."""
    hg = _host_graph(form, "float")
    g = _wgraph(mem, hg, "float")

    def steps():
        rfd = pg.get_objective(mem, g, pg.OBJ_WMOD)
        part = np.arange(g.n, dtype=np.int32)
        l0 = _lib.lib().pggc_launch_count()
        pg.local_move(mem, g, part, rfd, True)
        launches = _lib.lib().pggc_launch_count() - l0
        vcmap, nc = pg.coarsen_leidenR(mem, g, part, rfd, 11, 5)
        first = part.copy()
        pg.local_move_strict(mem, g, part, rfd, False)
        coarse = pg.build_coarse_graph(mem, g, vcmap, nc).to_host()
        return launches, [first, part, vcmap, nc, rfd.obj, rfd.total_deg(), *coarse]

    steps()  # the products kept with the graph
    one_launch, want = steps()
    _lib.check(_lib.lib().pggc_debug_set_cluster_limit(mem.handle, blocks))
    try:
        launches, got = steps()
    finally:
        _lib.check(_lib.lib().pggc_debug_set_cluster_limit(mem.handle, 16))
    assert (launches > one_launch) == (blocks < 8)
    for x, y in zip(got, want):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("strict", [False, True])
@pytest.mark.parametrize("form,weights", [("one_vertex", None), ("classes_0_to_3", "float"), ("move_16k", None),
                                          ("steps_40k", "float"), ("steps_40k", None), ("steps_hubs", "int")])
def test_profile_counts_the_same_bytes(mem, form, weights, strict):
    """The algorithmic bytes of a local move do not depend on the path that runs it."""
    hg = _host_graph(form, weights)
    g = _wgraph(mem, hg, weights)
    ct = _lib.ctypes

    def counted():
        rfd = pg.get_objective(mem, g, _objective(weights))
        part = np.arange(g.n, dtype=np.int32)
        pg.local_move(mem, g, part, rfd, True, sweep_limit=-1 if strict else 2)
        _lib.check(_lib.lib().pggc_profile_reset(mem.handle))
        _lib.check(_lib.lib().pggc_profile_enable(mem.handle, 1))
        try:
            (pg.local_move_strict if strict else pg.local_move)(mem, g, part, rfd, False)
        finally:
            _lib.check(_lib.lib().pggc_profile_enable(mem.handle, 0))
        out = {}
        for f in ("select_warp", "select_block", "select_huge", "afterburner_warp", "own_weights", "step_select",
                  "step_afterburner", "step_own", "local_move_small"):
            launches, ms, nbytes = ct.c_int64(), ct.c_double(), ct.c_double()
            _lib.check(_lib.lib().pggc_profile_read(mem.handle, f.encode(), ct.byref(launches), ct.byref(ms),
                                                    ct.byref(nbytes)))
            out[f] = (launches.value, nbytes.value)
        return out

    got = counted()
    with general_path(mem):
        want = counted()
    if strict and got["select_warp"][0]:
        return  # candidates: the one-launch sweep came before the general path's
    assert got["select_warp"][0] == 0 and want["local_move_small"][0] == want["step_select"][0] == 0
    assert sum(b for _, b in got.values()) == sum(b for _, b in want.values()) > 0


def _one_feature(f, sign):
    """A network whose logit is sign * feature f."""
    p = np.zeros(M.N_PARAMS, np.float32)
    p[M.O_W1 + f], p[M.O_W1 + 8 + f] = sign, -sign
    p[M.O_W2], p[M.O_W2 + 32 + 1] = 1, 1
    p[M.O_W3], p[M.O_W3 + 1] = 1, -1
    return p


# networks that reject some vertices: by the share of weight inside, the last gain, having moved in the last sweep,
# the size and the volume of the cluster, the sweep's number, and by all features at once
NETS = {"inside": (_one_feature(1, -1), -0.6), "gain": (_one_feature(2, -1), -0.1), "moved": (_one_feature(3, -1), -0.5),
        "size": (_one_feature(4, -1), -0.2), "volume": (_one_feature(5, -1), None), "sweep": (_one_feature(7, -1), -0.3),
        "all": (M.init_params(3), 0.05)}


@pytest.mark.parametrize("net", list(NETS))
@pytest.mark.parametrize("form,weights", [("classes_0_to_3", "float"), ("move_16k", None), ("steps_40k", "float"),
                                          ("steps_hubs", None)])
def test_filtered_moves(mem, form, weights, net):
    """The filter's features and counts are those of the class kernels: the same vertices are skipped."""
    hg = _host_graph(form, weights)
    g = _wgraph(mem, hg, weights)
    params, threshold = NETS[net]
    if threshold is None:
        threshold = -6.0 / g.n  # six vertices' share of the volume

    def run():
        MF.enable(mem, params, threshold)
        MF.stats(mem, reset=True)
        try:
            rfd = pg.get_objective(mem, g, _objective(weights))
            part = np.arange(g.n, dtype=np.int32)
            out = []
            for initial in (True, False):
                st = pg.local_move(mem, g, part, rfd, initial)
                out.append((part.copy(), st["sweeps"], st["moves"], rfd.obj, *MF.stats(mem)))
            rfd = pg.get_objective(mem, g, _objective(weights))
            labels, st = pg.run_clustering(mem, g, rfd, method=pg.METHOD_LEIDEN_PLUS, ex_iters=0, seed=9)
            out.append((labels, *st.values(), *MF.stats(mem)))
        finally:
            MF.disable(mem)
        return out

    got = run()
    with general_path(mem):
        want = run()
    for a, b in zip(got, want):
        for x, y in zip(a, b):
            np.testing.assert_array_equal(x, y)
    evaluated, skipped = got[1][-2:]
    assert evaluated > 0 and skipped > 0


@pytest.mark.parametrize("n,d,fits", [(11702, 10, True), (11703, 10, False),  # edges plus four a vertex: 163,840
                                      (2114, 62, True), (2115, 62, False),    # 131,072 edges
                                      (3072, 64, True), (3073, 64, False)])   # long rows: 196,608 edges
def test_size_limits_of_the_one_launch_move(mem, n, d, fits):
    """Rings where every vertex has d neighbours, at the limits and just above: the path that runs, and its answer."""
    col = np.sort((np.arange(n)[:, None] + np.delete(np.arange(-(d // 2), d // 2 + 1), d // 2)) % n, axis=1)
    g = pg.weighted_graph(mem, np.arange(n + 1, dtype=np.int64) * d, col.astype(np.int32).ravel(), None,
                          objective=pg.OBJ_MOD)

    def move():
        rfd = pg.get_objective(mem, g, pg.OBJ_MOD)
        part = np.arange(n, dtype=np.int32)
        l0 = _lib.lib().pggc_launch_count()
        st = pg.local_move(mem, g, part, rfd, True)
        return _lib.lib().pggc_launch_count() - l0, (part, st["sweeps"], st["moves"], rfd.obj)

    move()  # the products kept with the graph
    launches, got = move()
    assert (launches <= 3) == fits  # label check and move
    with general_path(mem):
        _, want = move()
    for x, y in zip(got, want):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("weights", [None, "int", "float"])
@pytest.mark.parametrize("n,d,nc,one", [(8000, 10, 1025, True), (8000, 10, 5000, True), (8200, 10, 1025, False),
                                        (24000, 6, 20000, True), (24600, 6, 1100, False),
                                        (1200, 64, 1030, True), (1200, 66, 1030, False),   # degree limit of the lists
                                        (1200, 66, 1024, True)])                           # the matrix has none here
def test_which_contraction_runs(mem, n, d, nc, one, weights):
    """Rings of even degree around the limits, one cluster of a third of the vertices: the path, and its rows."""
    col = np.sort((np.arange(n)[:, None] + np.delete(np.arange(-(d // 2), d // 2 + 1), d // 2)) % n, axis=1).ravel()
    src = np.repeat(np.arange(n), d)
    w = None
    if weights:
        k = (np.minimum(src, col) * n + np.maximum(src, col)) * 2654435761 % 1000003
        w = (k % 9 - 2).astype(np.int32) if weights == "int" else ((k + 1) * 2.0 ** -20).astype(np.float32)
    g = pg.weighted_graph(mem, np.arange(n + 1, dtype=np.int64) * d, col.astype(np.int32), w,
                          objective=_objective(weights))
    rng = np.random.default_rng(nc)
    rest = n - nc
    m = np.concatenate([np.arange(nc), np.where(rng.random(rest) < 0.33, 0, rng.integers(0, nc, rest))])
    vcmap = rng.permutation(m).astype(np.int32)
    # the degrees are known from an earlier move
    pg.local_move(mem, g, np.arange(n, dtype=np.int32), pg.get_objective(mem, g, _objective(weights)), True)
    l0 = _lib.lib().pggc_launch_count()
    got = pg.build_coarse_graph(mem, g, vcmap, nc)
    launches = _lib.lib().pggc_launch_count() - l0
    assert (launches <= 4) == one  # label check, contraction, vertex weights
    with general_path(mem):
        want = pg.build_coarse_graph(mem, g, vcmap, nc)
    for a, b in zip(got.to_host(), want.to_host()):
        assert np.array_equal(a, b)


def test_contraction_of_a_skewed_graph_is_general(mem):
    """A hub's row would be a few lanes' work: 8,193 edges go to the general path also with few clusters."""
    for leaves, one in ((8192, True), (8193, False)):
        g = pg.graph_from_edges(mem, leaves + 1, np.zeros(leaves, np.int32), np.arange(1, leaves + 1, dtype=np.int32))
        vcmap = (np.arange(leaves + 1) % 11).astype(np.int32)
        pg.generate_orderings(mem, g)
        pg.local_move(mem, g, np.arange(g.n, dtype=np.int32), pg.get_objective(mem, g, pg.OBJ_MOD), True)
        l0 = _lib.lib().pggc_launch_count()
        c = pg.build_coarse_graph(mem, g, vcmap, 11)
        assert (_lib.lib().pggc_launch_count() - l0 <= 4) == one
        rowptr, col, w, _ = c.to_host()
        hub = [(leaves + 1 - k + 10) // 11 for k in range(1, 11)]  # leaves in the other clusters, all joined to vertex 0
        assert np.array_equal(rowptr, np.concatenate([[0, 10], 10 + np.arange(1, 11)]))
        assert np.array_equal(col, np.concatenate([np.arange(1, 11), np.zeros(10)]))
        assert np.array_equal(w, hub + hub)
