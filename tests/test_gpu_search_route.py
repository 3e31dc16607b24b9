"""Which search runs a call: the profile sweep by default, the tree search where
an option of the tree asks for it, and the tree search after the sweep where its
grid cannot hold the domain. Results are the same on every route; without these
tests a sweep that turned every call down would pass the tests that compare it
with the tree."""
import ctypes as C

import numpy as np
import pytest

from horayzon_extpar_gb300 import _lib, horizon_svf_comp_py, synthetic
from horayzon_extpar_gb300.horizon_svf import horizon_svf_comp_batch

pytestmark = pytest.mark.gpu

ARGS = (24, 1, 40000.0, 0.2, 1, 2)


def _run(inputs, args=ARGS, **kw):
    h, s, st = horizon_svf_comp_py(*inputs, *args, return_stats=True, **kw)
    return h, s, st["num_rays"], st["search"]


def _same(inputs, search, args=ARGS, **kw):
    h0, s0, n0, by0 = _run(inputs, args, leaf_size=2, **kw)
    h1, s1, n1, by1 = _run(inputs, args, **kw)
    assert by0 == "tree" and by1 == search
    np.testing.assert_array_equal(h1, h0)
    np.testing.assert_array_equal(s1, s0)
    assert n1 == n0


@pytest.mark.parametrize("dkw,args,kw", [
    (dict(edge_km=1.0, box_km=4.0, seed=1), ARGS, {}),
    (dict(edge_km=0.1, box_km=8.0, seed=3, kind="eroded", hmin=0.0, hmax=3000.0),
     (37, 1, 8000.0, 0.2, 1, 1), {}),
    (dict(edge_km=0.1, box_km=5.0, seed=4, kind="eroded", hmin=0.0, hmax=2500.0),
     (24, 0, 15000.0, 2.0, 2, 2), {"precision": 1}),
    (dict(edge_km=40.0, box_km=2000.0, seed=5, hmax=6000.0, lat0_deg=70.0),
     (24, 1, 500000.0, 0.2, 1, 2), {}),
    (dict(edge_km=2.5, box_km=80.0, seed=8), ARGS, {"elev_floor_deg": 7.3}),
    (dict(edge_km=0.5, box_km=95.0, seed=10, hmax=3000.0), (45, 1, 6000.0, 0.2, 2, 0),
     {"cells": (3001, 14003)}),
])
def test_defaults_run_the_sweep(dkw, args, kw):
    _same(synthetic.make_domain(**dkw).inputs(), "sweep", args, **kw)


def test_a_batch_runs_the_sweep():
    doms = [(d.inputs(), a) for d, a in synthetic.make_batch(n_domains=3, seed=3, min_cells=300,
                                                             max_cells=3000)]
    assert horizon_svf_comp_batch(doms, return_stats=True)[1]["search"] == "sweep"
    assert horizon_svf_comp_batch(doms, return_stats=True, leaf_size=2)[1]["search"] == "tree"


@pytest.mark.parametrize("kw", [
    {"kernel": _lib.HZ_KERNEL_PER_CELL}, {"kernel": _lib.HZ_KERNEL_PERSISTENT_BVH2},
    {"count_work": True}, {"elev_walk": 1}, {"advance_min": 16}, {"leaf_min": 1}, {"leaf_size": 4},
    {"queue_chunk": 32}, {"bvh_treelets": True}, {"occluder_cache": False}])
def test_options_of_the_tree_run_the_tree(kw):
    d = synthetic.make_domain(edge_km=2.5, box_km=30.0, seed=2)
    assert _run(d.inputs(), **kw)[3] == "tree"


def test_a_wide_domain_falls_back():
    d = synthetic.make_domain(edge_km=2.0, box_km=20.0, seed=13)
    inputs = [np.array(a) for a in d.inputs()]
    half = d.ncell // 2
    inputs[0][half:] += 2.0  # 115 degrees: the mean direction shows it
    _same(inputs, "sweep, then tree", (12, 1, 20000.0, 0.2, 1, 2))
    inputs[0][half:] -= 0.7  # 75 degrees: the grid's bounds do
    _same(inputs, "sweep, then tree", (12, 1, 20000.0, 0.2, 1, 2))


def test_lists_beyond_their_capacity_fall_back():
    """Triangles two to three cells across, twenty layers of them: more entries than
    twelve per triangle, which the lists have room for."""
    from scipy.spatial import cKDTree
    d = synthetic.make_domain(edge_km=1.0, box_km=40.0, seed=21)
    clon, clat, h, vlon, vlat, cov = (np.array(a) for a in d.inputs())
    scale = np.cos(vlat.mean())
    tree = cKDTree(np.stack([clon * scale, clat], 1))
    ring = 2.6 / 6371.0
    full = np.nonzero((cov != -2).all(axis=0))[0]
    for k in range(6):
        t = np.pi / 3 * k
        at = np.stack([vlon[full] * scale + ring * np.sin(t), vlat[full] + ring * np.cos(t)], 1)
        cov[k, full] = tree.query(at)[1]
    distinct = np.sort(cov[:, full], axis=0)
    cov[:, full[(distinct[1:] == distinct[:-1]).any(axis=0)]] = -2  # rings cut by the border
    _same((clon, clat, h, vlon, vlat, cov), "sweep, then tree", (4, 1, 2000.0, 0.2, 1, 2))


def test_a_failed_call_reports_no_search():
    d = synthetic.make_domain(edge_km=2.5, box_km=30.0, seed=2)
    _run(d.inputs())
    assert _lib.load().hz_last_search() == 1
    h = np.empty(4)
    p = h.ctypes.data_as(C.POINTER(C.c_double))
    i = np.empty(4, dtype=np.int32).ctypes.data_as(C.POINTER(C.c_int32))
    assert _lib.load().hz_horizon_svf(p, p, p, p, p, i, p, p, 0, 0, 24, 1, 4e4, 0.2, 1, 2, None,
                                      None) == _lib.HZ_ERR_VALUE
    assert _lib.load().hz_last_search() == 0


@pytest.mark.parametrize("dkw,dist,elev,search", [
    # 11,000 cells and more: up to 0.03 of the search radius, and to 5 km
    (dict(edge_km=1.0, box_km=75.0, seed=31), 20000.0, 600.0, "sweep"),
    (dict(edge_km=1.0, box_km=75.0, seed=31), 20000.0, 601.0, "tree"),
    (dict(edge_km=10.0, box_km=750.0, seed=32), 400000.0, 5000.0, "sweep"),
    (dict(edge_km=10.0, box_km=750.0, seed=32), 400000.0, 5001.0, "tree"),
    (dict(edge_km=2.5, box_km=180.0, seed=34), 1000.0, 500.0, "tree"),
    # a few cells: beyond a tenth of the radius from above 5 km only
    (dict(edge_km=1.0, box_km=40.0, seed=33), 20000.0, 5000.0, "sweep"),
    (dict(edge_km=1.0, box_km=40.0, seed=33), 49000.0, 5001.0, "tree"),
    (dict(edge_km=1.0, box_km=40.0, seed=33), 60000.0, 5500.0, "sweep"),
])
def test_high_origins_run_the_tree(dkw, dist, elev, search):
    """Where the tree search is the faster one (many times at a tenth of the radius
    and 400,000 cells). With few cells traced the sweep runs again."""
    d = synthetic.make_domain(**dkw)
    args = (4, 1, dist, elev, 1, 2)
    h0, s0, n0, by = _run(d.inputs(), args)
    assert by == search
    h1, s1, n1, by = _run(d.inputs(), args, **({} if by == "tree" else {"leaf_size": 2}))
    assert by == "tree" and n1 == n0
    np.testing.assert_array_equal(h1, h0)
    np.testing.assert_array_equal(s1, s0)
    if elev < 5000.0:
        assert _run(d.inputs(), args, cells=(500, 3000))[3] == "sweep"


def _holes(d, share):
    inputs = [np.array(a) for a in d.inputs()]
    inputs[5][:, np.random.default_rng(1).random(d.nvertex) < share] = -2
    return tuple(inputs)


@pytest.mark.parametrize("share,grid_type,search", [
    (0.0, 1, "sweep"), (0.1, 1, "sweep"), (0.1, 0, "sweep"), (0.3, 1, "sweep, then tree"),
    (0.3, 0, "sweep, then tree")])
def test_meshes_with_many_holes_run_the_tree(share, grid_type, search):
    """59,000 cells, 30,000 ICON vertices: a tenth of them missing is repaired, of a third
    the tree search is the faster one; a range of the cells has its share of them."""
    d = synthetic.make_domain(edge_km=0.2, box_km=32.0, seed=41)
    inputs, args = _holes(d, share), (4, grid_type, 3000.0, 0.2, 1, 2)
    _same(inputs, search, args)
    if share == 0.3 and grid_type == 1:
        _same(inputs, "sweep", args, cells=(20000, 40000))


@pytest.mark.parametrize("grid_type", [0, 1])
def test_a_domain_without_triangles_in_parts_runs_the_sweep(grid_type):
    """Only the south-west third of the vertices has its triangles: the triangles that
    the cells lack are as many as with a third of the vertices missing, the cells
    at an edge of the mesh are few."""
    d = synthetic.make_domain(edge_km=0.2, box_km=32.0, seed=41)
    inputs = [np.array(a) for a in d.inputs()]
    lon, lat = inputs[3], inputs[4]
    outside = ((lon - lon.min()) / np.ptp(lon) > 0.58) | ((lat - lat.min()) / np.ptp(lat) > 0.58)
    inputs[5][:, outside] = -2
    _same(inputs, "sweep", (4, grid_type, 3000.0, 0.2, 1, 2))


def test_holes_of_a_batch_add_up():
    d = synthetic.make_domain(edge_km=0.2, box_km=32.0, seed=41)
    one = (_holes(d, 0.1), (4, 1, 3000.0, 0.2, 1, 2))
    for n, search in ((2, "sweep"), (4, "sweep, then tree")):
        outs, st = horizon_svf_comp_batch([one] * n, return_stats=True)
        assert st["search"] == search
        tree = horizon_svf_comp_batch([one] * n, leaf_size=2)
        assert all(np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
                   for a, b in zip(outs, tree))


def _beside(a, b):
    """Two domains as one mesh without a triangle between them."""
    n = a[0].size
    return tuple(np.concatenate([x, y]) for x, y in zip(a[:5], b[:5])) + (
        np.ascontiguousarray(np.concatenate([a[5], np.where(b[5] == -2, -2, b[5] + n)], 1)),)


@pytest.mark.parametrize("deg,search", [(3, "sweep"), (20, "sweep, then tree"),
                                        (40, "sweep, then tree")])
def test_patches_far_apart_run_the_tree(deg, search):
    """The grid spans the gap: its cells hold 12 triangles at 3 degrees, 380 at 20."""
    a, b = ([np.array(x) for x in
             synthetic.make_domain(edge_km=1.0, box_km=60.0, seed=s).inputs()] for s in (5, 6))
    for k in (0, 3):
        b[k] += np.radians(deg)
        b[k + 1] += np.radians(deg / 2)
    _same(_beside(a, b), search, (4, 1, 20000.0, 0.2, 1, 2))


@pytest.mark.parametrize("ratio,search", [(10, "sweep"), (60, "sweep, then tree")])
def test_fine_patches_beside_coarse_ones_run_the_tree(ratio, search):
    """0.2 km cells beside cells 10 and 60 times as wide, the grid's cells between them."""
    a = [np.array(x) for x in
         synthetic.make_domain(edge_km=0.2, box_km=20.0, seed=7).inputs()]
    b = [np.array(x) for x in
         synthetic.make_domain(edge_km=0.2 * ratio, box_km=5.0 * ratio, seed=8).inputs()]
    east = (a[0].max() - b[0].min()) * 1.001
    b[0] += east
    b[3] += east
    _same(_beside(a, b), search, (4, 1, 20000.0, 0.2, 1, 2))


def test_vertices_that_join_far_cells_run_the_tree_at_once():
    """Every triangle spans much of the domain: going through all grid cells of each
    took the square of the mesh's size before the lists overflowed (here 40 ms, a
    minute for a million cells)."""
    d = synthetic.make_domain(edge_km=1.0, box_km=110.0, seed=15)
    inputs = [np.array(a) for a in d.inputs()]
    rng = np.random.default_rng(15)
    full = np.nonzero((inputs[5] != -2).all(axis=0))[0]
    for k in range(6):  # a cell per sextant of the domain: six different ones
        part = np.arange(k * (d.ncell // 6), (k + 1) * (d.ncell // 6))
        inputs[5][k, full] = rng.choice(part, full.size)
    args, kw = (4, 1, 20000.0, 0.2, 1, 2), dict(cells=(0, 64))
    _same(inputs, "sweep, then tree", args, **kw)

    def lost():
        st = horizon_svf_comp_py(*inputs, *args, return_stats=True, **kw)[2]
        return st["ms_total"] - sum(st[k] for k in ("ms_h2d", "ms_mesh", "ms_bvh", "ms_trace",
                                                    "ms_d2h"))

    assert min(lost() for _ in range(3)) < 10.0


def test_occluder_cache_of_the_tree_search_in_a_batch():
    """Both settings on the 4-wide tree (the default with the cache on is the sweep)."""
    doms = [(d.inputs(), a) for d, a in synthetic.make_batch(n_domains=3, seed=5, min_cells=300,
                                                             max_cells=3000)]
    off, st0 = horizon_svf_comp_batch(doms, leaf_size=2, occluder_cache=False, return_stats=True)
    on, st1 = horizon_svf_comp_batch(doms, leaf_size=2, return_stats=True)
    assert st0["search"] == st1["search"] == "tree" and st0["num_rays"] == st1["num_rays"]
    assert all(np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
               for a, b in zip(off, on))
