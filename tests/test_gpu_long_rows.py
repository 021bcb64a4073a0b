"""Rows and runs that one warp or block must not be left alone with: contraction
rows split across blocks, CSR validation and flattening by edge chunks, class
lists and row sums of graphs with hubs."""
import numpy as np
import pytest

import pennsylvaniagpugraphclustering_b200 as pg
from pennsylvaniagpugraphclustering_b200 import _lib
from pennsylvaniagpugraphclustering_b200 import move_filter as MF

pytestmark = pytest.mark.gpu


def _hub_graph(n, hubs, hub_deg, extra, gap, weights, seed):
    """Random pairs above a run of `gap` vertices without edges, and `hubs` hubs."""
    rng = np.random.default_rng(seed)
    u = np.concatenate([np.repeat(gap + np.arange(hubs), hub_deg), rng.integers(gap, n, extra)])
    v = np.concatenate([rng.integers(gap, n, hubs * hub_deg), rng.integers(gap, n, extra)])
    keep = u != v
    key = np.unique(np.concatenate([u[keep] * n + v[keep], v[keep] * n + u[keep]]).astype(np.int64))
    src, dst = key // n, key % n
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.int64)
    w = None
    if weights:
        lo, hi = np.minimum(src, dst), np.maximum(src, dst)
        _, inv = np.unique(lo * n + hi, return_inverse=True)
        if weights == "float":
            w = (0.5 + rng.integers(0, 1 << 24, inv.max() + 1) * 2.0 ** -24).astype(np.float32)[inv]
        else:
            w = rng.integers(-(1 << 30), 1 << 30, inv.max() + 1).astype(np.int32)[inv]  # sums leave 32 bits
    return rowptr, src, dst.astype(np.int32), w


# clusters: few long rows; rows with more keys than the shared table; one long row among many short ones
@pytest.mark.parametrize("weights", [None, "int", "float"])
@pytest.mark.parametrize("nc,share", [(1, 0.0), (3, 0.0), (700, 0.0), (9000, 0.0), (30000, 0.6)])
def test_contraction_of_long_rows(mem, nc, share, weights):
    n = 70001
    rowptr, src, col, w = _hub_graph(n, 4, 30000, 500000, 3000, weights, 7)
    rng = np.random.default_rng(nc)
    m = np.where(rng.random(n) < share, 0, rng.integers(0, nc, n))
    m[:nc] = np.arange(nc)
    vcmap = rng.permutation(m).astype(np.int32)
    objective = pg.OBJ_WMOD if weights else pg.OBJ_MOD
    g = pg.weighted_graph(mem, rowptr, col, w, objective=objective)
    crow, ccol, cw, _ = pg.build_coarse_graph(mem, g, vcmap, nc).to_host()
    a, b = vcmap[src].astype(np.int64), vcmap[col].astype(np.int64)
    keep = a != b
    key, inv = np.unique(a[keep] * nc + b[keep], return_inverse=True)
    wide = np.float64 if weights == "float" else np.int64
    vals = np.ones(len(src), wide) if w is None else w.astype(wide)
    total = np.zeros(len(key), wide)
    np.add.at(total, inv, vals[keep])
    assert np.array_equal(crow, np.concatenate([[0], np.cumsum(np.bincount(key // nc, minlength=nc))]))
    assert np.array_equal(ccol, key % nc)
    assert np.array_equal(cw, total.astype(np.float32 if weights == "float" else np.int32))


def _create(mem, rowptr, col):
    return pg.weighted_graph(mem, rowptr, col, None, objective=pg.OBJ_MOD)


@pytest.mark.parametrize("where", ["first", "chunk_end", "chunk_start", "hub", "last"])
@pytest.mark.parametrize("fault", ["loop", "range", "negative"])
def test_validation_finds_faults_anywhere(mem, where, fault):
    """One bad column; edges are checked 1,024 to a warp."""
    n = 9000
    rowptr, src, col, _ = _hub_graph(n, 2, 5000, 8000, 700, None, 3)
    _create(mem, rowptr, col)
    j = {"first": 0, "chunk_end": 1023, "chunk_start": 2048, "hub": int(rowptr[700]) + 3000, "last": len(col) - 1}[where]
    bad = col.copy()
    bad[j] = {"loop": src[j], "range": n, "negative": -1}[fault]
    with pytest.raises(_lib.InvalidArgument):
        _create(mem, rowptr, bad)


def test_local_move_with_hubs_matches_a_run_from_the_same_state(mem):
    """Hub movers are marked by blocks, the others by warps: the sweeps leave consistent own-cluster weights, so a
    second local move from the result reports the objective of the labels (above the launch-per-step size)."""
    n = (1 << 20) + 77
    rowptr, src, col, _ = _hub_graph(n, 5, 40000, 2000000, 1000, None, 11)
    g = _create(mem, rowptr, col)
    rfd = pg.get_objective(mem, g, pg.OBJ_MOD)
    part = np.arange(n, dtype=np.int32)
    pg.local_move(mem, g, part, rfd, True)
    assert rfd.get_objective() == pytest.approx(pg.verify_objective(mem, g, part)[0], rel=1e-12)
    pg.local_move(mem, g, part, rfd, False)
    assert rfd.get_objective() == pytest.approx(pg.verify_objective(mem, g, part)[0], rel=1e-12)
    deg = np.diff(rowptr)
    o1, _, off = pg.generate_orderings(mem, g)
    bucket = np.where(deg < 128, 0, np.where(deg < 15000, 1, 2))
    assert np.array_equal(o1, np.argsort(bucket, kind="stable"))


def _float_graph(n, seed, make):
    """A graph of dense rows (every select and contraction table) with the weights `make` draws."""
    rng = np.random.default_rng(seed)
    u = np.concatenate([rng.integers(0, n, n * 60), np.repeat(np.arange(6), 3000)])
    v = np.concatenate([rng.integers(0, n, n * 60) // 2, rng.integers(0, n, 18000)])
    keep = u != v
    key = np.unique(np.concatenate([u[keep] * n + v[keep], v[keep] * n + u[keep]]).astype(np.int64))
    src, dst = key // n, key % n
    lo, hi = np.minimum(src, dst), np.maximum(src, dst)
    _, inv = np.unique(lo * n + hi, return_inverse=True)
    w = make(rng, inv.max() + 1).astype(np.float32)[inv]
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.int64)
    return rowptr, src, dst.astype(np.int32), w


# whole units of 2^-24; the most fraction bits that units have, with a total below and above 2^52 of them; more
# bits than that (FP64 tables); zeros; negative weights, which have no units
UNIT_WEIGHTS = {
    "grid_24": lambda r, k: 0.5 + r.integers(0, 1 << 24, k) * 2.0 ** -24,
    "bits_40": lambda r, k: r.integers(1, 4, k) * 2.0 ** -40,
    "bits_40_large_total": lambda r, k: np.where(r.random(k) < 0.5, 2.0 ** -40, 0.25),
    "bits_41": lambda r, k: r.integers(1, 4, k) * 2.0 ** -41,
    "zeros": lambda r, k: r.integers(0, 2, k) * 0.75,
    "negative": lambda r, k: r.integers(-1, 4, k) * 0.5,
}


@pytest.mark.parametrize("n", [3001, 40001])
@pytest.mark.parametrize("kind", list(UNIT_WEIGHTS))
def test_float_tables_in_units(mem, kind, n):
    """Contraction against numpy sums (exact: every sum is a multiple of one power of two below 2^53 of them), and one
    select pass against sums per neighbour cluster."""
    rowptr, src, col, w = _float_graph(n, 5, UNIT_WEIGHTS[kind])
    g = pg.weighted_graph(mem, rowptr, col, w, objective=pg.OBJ_WMOD)
    for nc in (40, 1500):
        vcmap = np.random.default_rng(nc).permutation(np.arange(n) % nc).astype(np.int32)
        crow, ccol, cw, _ = pg.build_coarse_graph(mem, g, vcmap, nc).to_host()
        a, b = vcmap[src].astype(np.int64), vcmap[col].astype(np.int64)
        keep = a != b
        key, inv = np.unique(a[keep] * nc + b[keep], return_inverse=True)
        total = np.zeros(len(key))
        np.add.at(total, inv, w[keep].astype(np.float64))
        assert np.array_equal(ccol, key % nc) and np.array_equal(cw, total.astype(np.float32))
    # every vertex's best cluster has its sum of weights as the gain when nothing is subtracted (lambda 0)
    nc = 300
    part = np.random.default_rng(1).permutation(np.arange(n) % nc).astype(np.int32)
    rfd = pg.get_objective(mem, g, pg.OBJ_LCC, 0.0)
    key, inv = np.unique(src * nc + part[col], return_inverse=True)
    sums = np.zeros(len(key))
    np.add.at(sums, inv, w.astype(np.float64))
    own = np.zeros(n)
    mine = key % nc == part[key // nc]
    own[(key // nc)[mine]] = sums[mine]
    rfd.set_state(nc, np.zeros(nc), 0.0)
    dest, gain, _ = pg.select_pass(mem, g, rfd, part, own, np.full(n, -1, np.int32), 0.0, False)
    best = np.full(n, -np.inf)
    np.maximum.at(best, (key // nc)[~mine], np.where(sums > 0, sums, -np.inf)[~mine].astype(np.float32))
    # the threshold: nothing below the own-cluster weight, and at least 0
    moves = (best >= np.maximum(own.astype(np.float32), 0)) & np.isfinite(best)
    assert np.array_equal(dest >= 0, moves)
    assert np.array_equal(gain[moves], (best[moves].astype(np.float32) - own[moves].astype(np.float32)))


@pytest.mark.parametrize("weights", [False, True])
@pytest.mark.parametrize("how", ["strict", "logging"])
def test_rows_of_more_edges_than_vertices(mem, how, weights):
    """Parallel edges: 80 triples a - b - c in 1,000 vertices, 1,100 edges from a to b and 1,200 from b to c.  From
    {a}, {b, c} every a moves; its neighbour b gains that row in own-cluster weight, and the objective kept by the
    sweeps must be the labels' own.  Few enough movers for their rows to be pushed, enough for the flags."""
    n, k, ab, bc = 1000, 80, 1100, 1200
    a = 3 * np.arange(k, dtype=np.int32)
    src = np.concatenate([np.repeat(a, ab), np.repeat(a + 1, bc)])
    dst = src + 1
    w = (1 + np.arange(len(src)) % 3).astype(np.int32) if weights else None
    objective = pg.OBJ_WMOD if weights else pg.OBJ_MOD
    g = pg.graph_from_edges(mem, n, src, dst, w, symmetric=True, objective=objective)
    assert np.diff(g.to_host()[0]).max() > n
    part = np.arange(n, dtype=np.int32)
    part[a + 2] = a + 1
    rfd = pg.get_objective(mem, g, objective)
    td = np.zeros(n, np.int64)
    np.add.at(td, part, g.to_host()[3])
    rfd.set_state(n, td, 2.0 * (np.ones(len(src)) if w is None else w)[k * ab:].sum())
    if how == "strict":
        st = pg.local_move_strict(mem, g, part, rfd, False)
    else:
        MF.log_start(mem, 1 << 16)
        try:
            st = pg.local_move(mem, g, part, rfd, False, enable_simulated_annealing=False)
        finally:
            MF.log_stop(mem, 1 << 16)
    assert st["moves"] == k and np.array_equal(part[a], part[a + 1]) and np.array_equal(part[a], part[a + 2])
    assert rfd.get_objective() == pytest.approx(pg.verify_objective(mem, g, part, objective)[0], rel=1e-12)


@pytest.mark.parametrize("weights", [None, "int", "float"])
def test_contraction_at_the_long_row_limit(mem, weights):
    """Rows of exactly 131,072 member edges (a block's), just above (split across blocks), and of 80,000 with more
    distinct keys than the largest shared table (handed over by the block)."""
    d, n = 32, 120000
    u = np.repeat(np.arange(n), d)
    v = (u + np.tile(np.concatenate([np.arange(-16, 0), np.arange(1, 17)]) * 1201, n)) % n
    o = np.lexsort((v, u))
    src, col = u[o], v[o].astype(np.int32)
    w = None
    if weights:
        k = (np.minimum(src, col).astype(np.int64) * n + np.maximum(src, col)) * 2654435761 % 1000003
        w = (k % 9 - 2).astype(np.int32) if weights == "int" else ((k + 1) * 2.0 ** -20).astype(np.float32)
    g = pg.weighted_graph(mem, np.arange(n + 1, dtype=np.int64) * d, col, w,
                          objective=pg.OBJ_WMOD if weights else pg.OBJ_MOD)
    nc = 60003
    m = 3 + np.random.default_rng(1).permutation(np.arange(n) % (nc - 3))
    m[:4096] = 0
    m[50000:54097] = 1
    spread = np.arange(60000, n)[::24][:2500]
    m[spread] = 2
    vcmap = np.unique(m, return_inverse=True)[1].astype(np.int32)
    nc = int(vcmap.max()) + 1
    assert [d * int((vcmap == c).sum()) for c in range(3)] == [131072, 131104, 80000]
    crow, ccol, cw, _ = pg.build_coarse_graph(mem, g, vcmap, nc).to_host()
    a, b = vcmap[src].astype(np.int64), vcmap[col].astype(np.int64)
    keep = a != b
    key, inv = np.unique(a[keep] * nc + b[keep], return_inverse=True)
    assert np.sum(key // nc == 2) > 16384
    wide = np.float64 if weights == "float" else np.int64
    total = np.zeros(len(key), wide)
    np.add.at(total, inv, np.ones(int(keep.sum()), wide) if w is None else w[keep].astype(wide))
    assert np.array_equal(crow, np.concatenate([[0], np.cumsum(np.bincount(key // nc, minlength=nc))]))
    assert np.array_equal(ccol, key % nc)
    assert np.array_equal(cw, total.astype(np.float32 if weights == "float" else np.int32))


def test_validation_of_chunks_of_1024(mem):
    """Above 9.7 M edges a warp checks 1,024 of them (fewer in the smaller graphs above)."""
    d, n = 32, 330000
    off = np.concatenate([np.arange(-16, 0), np.arange(1, 17)])
    col = np.sort((np.arange(n)[:, None] + off) % n, axis=1).astype(np.int32).ravel()
    rowptr = np.arange(n + 1, dtype=np.int64) * d
    _create(mem, rowptr, col)
    for j in (0, 1023, 1024, 5 * 1024 * 1024 - 1, len(col) - 1):
        for fault in (j // d, n, -1):
            bad = col.copy()
            bad[j] = fault
            with pytest.raises(_lib.InvalidArgument):
                _create(mem, rowptr, bad)


@pytest.mark.parametrize("weights", ["float", "int"])
def test_rows_at_batch_edges_match_oracle(mem, weights):
    """Rows of up to, exactly and just above two, four and eight groups of 32 edges, and whole batches with every
    remainder, in the own-weight, afterburner and inner-connectivity sums of a run."""
    from oracle import oracle as O
    degs = [31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 159, 160, 161, 191, 193, 224, 255, 256, 257, 287, 320,
            352, 383, 385, 449, 511, 512, 513, 1023, 1025]
    n = 9000
    rng = np.random.default_rng(5)
    hubs = np.arange(len(degs)) * 7
    leaves = np.setdiff1d(np.arange(n), hubs)
    u = np.concatenate([np.repeat(h, k) for h, k in zip(hubs, degs)])
    # a hub's leaves come from its own stretch of the ring mostly
    v = np.concatenate([leaves[(np.arange(k) + i * 270) % len(leaves)] for i, k in enumerate(degs)])
    ring = np.arange(len(leaves))
    u = np.concatenate([u, leaves, leaves])
    v = np.concatenate([v, leaves[(ring + 1) % len(leaves)], leaves[(ring + 2) % len(leaves)]])
    key = np.unique(np.concatenate([u * n + v, v * n + u]).astype(np.int64))
    src, col = key // n, (key % n).astype(np.int32)
    deg = np.bincount(src, minlength=n)
    assert np.array_equal(deg[hubs], degs)
    lo, hi = np.minimum(src, col), np.maximum(src, col)
    _, inv = np.unique(lo * n + hi, return_inverse=True)
    k = rng.integers(1, 1 << 22, int(inv.max()) + 1)[inv]
    w = (k * 2.0 ** -22).astype(np.float32) if weights == "float" else (1 + k % 5).astype(np.int32)
    rowptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
    g = pg.weighted_graph(mem, rowptr, col, w, objective=pg.OBJ_WMOD)
    og = O.Graph(rowptr, col, w, objective=pg.OBJ_WMOD)
    for seed in (1, 2):
        cd = pg.get_objective(mem, g, pg.OBJ_WMOD)
        lab, st = pg.run_clustering(mem, g, cd, method=pg.METHOD_LEIDEN_PLUS, ex_iters=1, seed=seed)
        lo_, so = O.run_clustering(og, O.ClusterData(og, pg.OBJ_WMOD, 1.0), method=pg.METHOD_LEIDEN_PLUS, ex_iters=1,
                                   seed=seed)
        assert np.array_equal(lab, lo_) and st["objective"] == so.objective
    # a run's FP32 coarse edges are sums rounded to 24 bits
    rel = 2.0 ** -23 if weights == "float" else 1e-12
    assert pg.verify_objective(mem, g, lab, pg.OBJ_WMOD)[0] == pytest.approx(st["objective"], rel=rel)
