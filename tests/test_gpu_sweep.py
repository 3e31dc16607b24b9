"""The profile sweep against the tree search: the same lattice rays decide, so
horizons, sky view factors and ray counts are the same bits. Cases at the edges
of its ranges: one triangle fan, no triangle, cells under and beside the mesh,
coarse grids whose search radius spans much of the domain, azimuth counts that
do not divide into the sweep's runs, floors, cell ranges, given starts, and
domains its grid cannot hold."""
import numpy as np
import pytest

from horayzon_extpar_gb300 import horizon_svf_comp_py, synthetic
from horayzon_extpar_gb300.horizon_svf import horizon_svf_comp_batch

pytestmark = pytest.mark.gpu


def _same(inputs, args, **kw):
    # An explicit tree option selects the tree search.
    h0, s0, st0 = horizon_svf_comp_py(*inputs, *args, return_stats=True, leaf_size=2, **kw)
    h1, s1, st1 = horizon_svf_comp_py(*inputs, *args, return_stats=True, **kw)
    assert np.array_equal(h0, h1, equal_nan=True)
    assert np.array_equal(s0, s1, equal_nan=True)
    assert st0["num_rays"] == st1["num_rays"]
    assert st0["n_tri"] == st1["n_tri"]
    return st0, st1


@pytest.mark.parametrize("dkw,args,kw", [
    # nearly every cell lies on the border and looks under the mesh's edge
    (dict(edge_km=1.0, box_km=4.0, seed=1), (24, 1, 40000.0, 0.2, 1, 2), {}),
    (dict(edge_km=1.0, box_km=6.0, seed=2), (7, 0, 1000.0, 0.1, 3, 0), {}),
    # steep, fine terrain; azimuths that do not divide into runs
    (dict(edge_km=0.1, box_km=8.0, seed=3, kind="eroded", hmin=0.0, hmax=3000.0),
     (37, 1, 8000.0, 0.2, 1, 1), {}),
    (dict(edge_km=0.1, box_km=5.0, seed=4, kind="eroded", hmin=0.0, hmax=2500.0),
     (24, 0, 15000.0, 2.0, 2, 2), {"precision": 1}),
    # coarse cells, a search radius of a quarter of the domain, high latitude
    (dict(edge_km=40.0, box_km=2000.0, seed=5, hmax=6000.0, lat0_deg=70.0),
     (24, 1, 500000.0, 0.2, 1, 2), {}),
    (dict(edge_km=10.0, box_km=900.0, seed=6, lat0_deg=-33.0, lon0_deg=151.0,
          face_rotation_deg=41.0), (48, 1, 100000.0, 0.2, 1, 0), {"precision": 1}),
    # flat terrain: horizons decided by the smallest differences
    (dict(edge_km=2.0, box_km=60.0, seed=7, hmin=100.0, hmax=100.0, n_features=0),
     (24, 1, 40000.0, 0.1, 1, 2), {}),
    # floors of the downward walk
    (dict(edge_km=2.5, box_km=80.0, seed=8), (24, 1, 40000.0, 0.2, 1, 2),
     {"elev_floor_deg": -0.25}),
    (dict(edge_km=2.5, box_km=80.0, seed=8), (24, 1, 40000.0, 0.2, 1, 2),
     {"elev_floor_deg": 7.3}),
    # a range of cells
    (dict(edge_km=1.0, box_km=40.0, seed=9), (24, 1, 20000.0, 0.2, 5, 1),
     {"cells": (1001, 1778)}),
    # cells enough for runs of several azimuths, shorter ones for the last cells
    (dict(edge_km=0.5, box_km=95.0, seed=10, hmax=3000.0), (77, 1, 6000.0, 0.2, 1, 2), {}),
    (dict(edge_km=0.5, box_km=95.0, seed=10, hmax=3000.0), (45, 1, 6000.0, 0.2, 2, 0),
     {"cells": (3001, 14003), "precision": 1}),
    # azimuths close together, and starts one step below the one before
    (dict(edge_km=0.5, box_km=40.0, seed=14, hmax=4000.0), (159, 1, 9000.0, 0.2, 1, 2), {}),
    (dict(edge_km=0.5, box_km=40.0, seed=14, hmax=4000.0), (80, 1, 9000.0, 0.2, 2, 1), {}),
    (dict(edge_km=0.2, box_km=8.0, seed=15, kind="eroded", hmax=3000.0),
     (360, 0, 8000.0, 0.2, 1, 2), {"precision": 1}),
    # a triangle cut by many rays at the search radius, beyond it at the higher
    (dict(edge_km=0.24629858041449693, box_km=17.611548057004665, kind="eroded",
          hmin=268.98230903271724, hmax=9000, hurst=0.9368420793831944, n_features=6, seed=319,
          lat0_deg=18.69738742425085, lon0_deg=-85.1331917032566, face_rotation_deg=0.0),
     (24, 1, 5000.0, 0.2, 1, 2), {}),
])
def test_gpu_sweep_is_the_tree_search(dkw, args, kw):
    d = synthetic.make_domain(**dkw)
    _same(d.inputs(), args, **kw)


def test_gpu_sweep_without_triangles_and_with_one_fan():
    d = synthetic.make_domain(edge_km=1.0, box_km=6.0, seed=11)
    cov = np.full_like(d.cells_of_vertex, -2)
    _same((*d.inputs()[:5], cov), (24, 1, 40000.0, 0.2, 1, 2))
    full = np.nonzero((d.cells_of_vertex != -2).all(axis=0))[0][0]
    cov[:, full] = d.cells_of_vertex[:, full]
    for gt in (0, 1):
        _same((*d.inputs()[:5], cov), (24, gt, 40000.0, 0.2, 1, 2))


def test_gpu_sweep_with_holes_and_spikes():
    """Patches of the mesh missing (rays pass under and through the edges) and
    single cells a kilometre above their neighbours."""
    d = synthetic.make_domain(edge_km=0.5, box_km=30.0, seed=12)
    rng = np.random.default_rng(12)
    clon, clat, h, vlon, vlat, cov = (np.array(a) for a in d.inputs())
    cov[:, rng.random(cov.shape[1]) < 0.1] = -2
    h[rng.random(h.size) < 0.01] += 1000.0
    for gt in (0, 1):
        _same((clon, clat, h, vlon, vlat, cov), (24, gt, 20000.0, 0.2, 1, 2))


def test_gpu_sweep_falls_back_on_wide_domains():
    """Cells around half the globe: the grid cannot hold them, the tree search
    runs in its place."""
    d = synthetic.make_domain(edge_km=2.0, box_km=30.0, seed=13)
    clon, clat, h, vlon, vlat, cov = (np.array(a) for a in d.inputs())
    n = clon.size // 2
    clon[n:] += 2.0  # the second half of the cells 115 degrees further east
    _same((clon, clat, h, vlon, vlat, cov), (12, 1, 20000.0, 0.2, 1, 2))
    clon[n:] -= 0.7  # 75 degrees: the mean direction does not show it
    _same((clon, clat, h, vlon, vlat, cov), (12, 1, 20000.0, 0.2, 1, 2))


def test_gpu_sweep_batch_of_unlike_domains():
    doms = [(synthetic.make_domain(edge_km=e, box_km=b, seed=s).inputs(),
             (nh, gt, dist, 0.2, rf, sv))
            for e, b, s, nh, gt, dist, rf, sv in
            [(2.5, 20.0, 21, 24, 1, 40000.0, 1, 2), (0.2, 12.0, 22, 5, 0, 3000.0, 1, 0),
             (1.0, 50.0, 23, 36, 1, 25000.0, 2, 1), (5.0, 300.0, 24, 16, 1, 90000.0, 1, 2)]]
    tree = horizon_svf_comp_batch(doms, leaf_size=2)
    for (h0, s0), (h1, s1) in zip(tree, horizon_svf_comp_batch(doms)):
        assert np.array_equal(h0, h1) and np.array_equal(s0, s1)


@pytest.mark.parametrize("groups,every", [(0, False), (4, False), (0, True)])
def test_gpu_sweep_given_starts(groups, every):
    torch = pytest.importorskip("torch")
    from horayzon_extpar_gb300 import horizon_svf_comp_device
    d = synthetic.make_domain(edge_km=0.2, box_km=12.0, seed=31, kind="eroded", hmax=2500.0)
    t = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in d.inputs()]
    args = (24, 1, 8000.0, 0.2, 2, 2)
    g = torch.Generator().manual_seed(5)
    start = torch.randint(-200, 200, (48, d.ncell), generator=g).to(torch.int16)
    start[:, ::3] = torch.randint(-4, 12, start[:, ::3].shape, generator=g).to(torch.int16)
    start = start.cuda()
    out = []
    for kw in ({"leaf_size": 2}, {}):
        raw = torch.empty((48, d.ncell), dtype=torch.int16, device="cuda")
        h, s, st = horizon_svf_comp_device(*t, *args, start_index=start, raw_index=raw,
                                           mlp_azimuth_groups=groups, mlp_every_azimuth=every, **kw)
        out.append((h, s, raw, st["num_rays"]))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    assert torch.equal(out[0][2], out[1][2]) and out[0][3] == out[1][3]


@pytest.mark.parametrize("dkw,nh,grid_type,cells", [
    (dict(edge_km=5.0, box_km=1400.0, seed=6, hmax=2000.0, kind="fbm_ridged"), 24, 1, (81000, 89000)),
    (dict(edge_km=5.0, box_km=1400.0, seed=6, hmax=2000.0, kind="fbm_ridged"), 36, 0, (69000, 77000)),
    (dict(edge_km=5.0, box_km=1500.0, seed=3, hmax=3500.0), 24, 1, (90000, 98000)),
])
def test_gpu_sweep_of_far_rays_in_mid_air(dkw, nh, grid_type, cells):
    """Origins 50 km over the terrain: the rays that a search casts below its
    horizon end in mid-air or meet terrain hundreds of kilometres away, where the
    bounds of a ray's height have to hold the cosine of the angle at the centre.
    The horizons there are clipped to 0: the unclipped indices are compared. (A
    range of cells: for more of them the tree search runs.)"""
    torch = pytest.importorskip("torch")
    from horayzon_extpar_gb300 import horizon_svf_comp_device
    d = synthetic.make_domain(**dkw)
    t = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in d.inputs()]
    out = []
    for opt in ({"leaf_size": 2}, {}):
        raw = torch.zeros((nh, d.ncell), dtype=torch.int16, device="cuda")
        _, s, st = horizon_svf_comp_device(*t, nh, grid_type, 500000.0, 50000.0, 1, 2,
                                           raw_index=raw, cells=cells, **opt)
        out.append((raw, s[cells[0]:cells[1]].clone(), st["num_rays"], st["search"]))
    assert out[1][3] == "sweep"
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    assert out[0][2] == out[1][2]


@pytest.mark.parametrize("nh,search", [(4, "sweep"), (24, "sweep, then tree")])
def test_gpu_sweep_under_a_roof(nh, search):
    """A basin under a second sheet of cells: every ray of a full turn hits there,
    and each azimuth starts where the last one ended, a turn of 720 elevations
    further. The elevations leave the table (four azimuths), and the sweep's
    16-bit codes (more than thirteen)."""
    d = synthetic.make_domain(edge_km=0.5, box_km=15.0, seed=17)
    clon, clat, h, vlon, vlat, cov = (np.array(a) for a in d.inputs())
    x = (clon - clon.mean()) * np.cos(clat.mean()) * 6371.0
    y = (clat - clat.mean()) * 6371.0
    r = np.sqrt(x * x + y * y)
    ground = 500.0 + 2500.0 * np.minimum(r / 6.0, 1.1) ** 4
    n = clon.size
    inputs = (np.concatenate([clon, clon]), np.concatenate([clat, clat]),
              np.concatenate([ground, np.full(n, 1500.0)]), np.concatenate([vlon, vlon]),
              np.concatenate([vlat, vlat]),
              np.ascontiguousarray(np.concatenate([cov, np.where(cov == -2, -2, cov + n)], 1)))
    st0, st1 = _same(inputs, (nh, 1, 20000.0, 0.2, 1, 2))
    assert st0["num_rays"] > 700 * nh * np.sum(r < 3.0)  # full turns
    assert st1["search"] == search


def test_gpu_sweep_latency_holds_repair_and_outputs():
    """A batch of meshes with holes, whose cells are repaired for most of the search:
    their domains are done at its end, not when the sweep's last item is."""
    batch = []
    for seed in (51, 52):
        d = synthetic.make_domain(edge_km=1.0, box_km=140.0, seed=seed)
        inputs = [np.array(a) for a in d.inputs()]
        inputs[5][:, np.random.default_rng(seed).random(d.nvertex) < 0.05] = -2
        batch.append((inputs, (24, 1, 40000.0, 0.2, 1, 2)))
    for _ in range(2):
        _, st = horizon_svf_comp_batch(batch, return_stats=True)
    assert st["search"] == "sweep"
    assert all(0.85 * st["ms_trace"] < t < 1.05 * st["ms_trace"] for t in st["latency_ms"]), st


def test_gpu_sweep_groups_of_a_large_batch():
    """From 60M evaluations on the domains complete in groups of a quarter of the
    work, in ascending order of their work; results are those of single calls."""
    edges, boxes = [0.5] * 9, [40.0, 45.0, 160.0, 170.0, 180.0, 190.0, 200.0, 210.0, 220.0]
    doms = [(synthetic.make_domain(edge_km=e, box_km=b, seed=60 + k).inputs(),
             (36, 1, 4000.0, 0.2, 1, 2)) for k, (e, b) in enumerate(zip(edges, boxes))]
    order = [4, 0, 8, 2, 6, 1, 7, 3, 5]
    outs, st = horizon_svf_comp_batch([doms[k] for k in order], return_stats=True)
    assert st["search"] == "sweep"
    lat = np.empty(9)
    lat[order] = st["latency_ms"]
    assert sum(d[0][0].size for d in doms) * 36 >= 6e7
    assert lat[0] < 0.4 * lat[8] and lat[4] < 0.7 * lat[8]
    assert (np.diff(lat) > -0.1 * lat[8]).all()  # in order, within a group close together
    rays = 0
    for k, (h, s) in zip(order, outs):
        h1, s1, st1 = horizon_svf_comp_py(*doms[k][0], *doms[k][1], return_stats=True)
        assert np.array_equal(h, h1) and np.array_equal(s, s1)
        rays += st1["num_rays"]
    assert rays == st["num_rays"]
