"""Workloads of the terrain-horizon / sky-view-factor library.

Each case is one call that a user of the library makes: the horizon angles and
the sky view factor of every cell of a regional ICON grid, through one of the
public entry points. The grid shapes and terrain recipes are those of the
repository's benchmark (2.5 km, 1 km, 500 m and 100 m spacing) and of its
tests; the arguments cover what EXTPAR passes (num_hori 24 and 48, refined
azimuths, both triangulations, the three SVF kinds) and what a verification
run passes (many azimuths, the precise frame).

A case's fields: ``entry`` (``device``: CUDA tensors in and out, ``host``: the
numpy drop-in, ``batch``: many domains in one host call, ``restart``: the
device call started from an earlier run's horizons), the grid (``edge_km``,
``box_km``, ``lat``, ``lon``, ``rot``), the terrain (``kind``, ``hmin``,
``hmax``) and the scalar arguments of the call.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from horayzon_extpar_gb300.horizon_svf import (horizon_svf_comp_batch, horizon_svf_comp_device,
                                               horizon_svf_comp_py)
from horayzon_extpar_gb300.synthetic import R_EARTH, icon_like_grid


def _case(name, entry, edge_km, box_km, kind, hmin, hmax, num_hori=24, grid_type=1,
          dist=40000.0, ray_org_elev=0.2, refine=1, svf_type=2, precise=False, lat=46.0, lon=8.0,
          rot=0.0, n_domains=1):
    return dict(name=name, entry=entry, edge_km=edge_km, box_km=box_km, kind=kind, hmin=hmin,
                hmax=hmax, num_hori=num_hori, grid_type=grid_type, dist=dist,
                ray_org_elev=ray_org_elev, refine=refine, svf_type=svf_type, precise=precise,
                lat=lat, lon=lon, rot=rot, n_domains=n_domains)


def listed():
    return [
        # A test-sized domain that already lies on the GPU: the smallest call
        # (about 500 cells); latency and launches.
        _case("tiny_device", "device", 2.5, 40.0, "fbm", 0.0, 3000.0),
        # A small limited-area domain through the numpy drop-in, as a script
        # that calls the reference's binding would run it (about 7,800 cells).
        _case("small_host", "host", 2.5, 150.0, "fbm", 0.0, 3000.0, lat=-41.3, lon=171.5, rot=37.0),
        # The 2.5 km regional domain of an operational limited-area model
        # (about 57,000 cells).
        _case("regional_2500m", "device", 2.5, 400.0, "fbm", 0.0, 3000.0),
        # The same domain after an update of its orography, started from the
        # horizons of the earlier run, azimuths spread over the GPU.
        _case("restart_2500m", "restart", 2.5, 400.0, "fbm", 0.0, 3000.0),
        # A verification run: one horizon per degree and the plain geometric
        # SVF with sin weighting on a kilometre-scale domain.
        _case("azimuths_360", "device", 1.0, 100.0, "ridged", 100.0, 4000.0, num_hori=360,
              svf_type=1, lat=61.0, lon=9.5, rot=71.0),
        # Triangulation from the cell centres alone, 48 sectors, a shorter
        # search radius, the pure geometric SVF.
        _case("grid_type0_1km", "device", 1.0, 251.0, "ridged", 0.0, 4500.0, num_hori=48,
              grid_type=0, dist=20000.0, ray_org_elev=0.5, svf_type=0, lat=39.7, lon=-106.0,
              rot=15.0),
        # The precise (local) frame on a 500 m domain.
        _case("precise_500m", "device", 0.5, 150.0, "ridged", 200.0, 4800.0, precise=True),
        # EXTPAR's sector means: every sector the mean of ten azimuths.
        _case("refine10_500m", "device", 0.5, 150.0, "ridged", 200.0, 4800.0, refine=10),
        # Many nests and regions of different size in one call, host arrays.
        _case("batch_host", "batch", 1.25, 160.0, "fbm", 0.0, 3500.0, n_domains=14),
        # The numpy drop-in on a large domain: host copies in and out included.
        _case("host_500m", "host", 0.5, 300.0, "ridged", 200.0, 4800.0),
        # The 500 m, 600 x 600 km benchmark domain (3.1M cells).
        _case("large_500m", "device", 0.5, 600.0, "ridged", 200.0, 4800.0),
        # Hectometric nest: 100 m spacing in high mountains (1.2M cells).
        _case("nest_100m", "device", 0.1, 75.0, "eroded", 500.0, 4200.0, lat=46.5, lon=8.3),
    ]


def draw(rng):
    entry = rng.choice(["device", "device", "device", "host", "host", "batch", "restart"])
    num_hori = rng.choice([rng.randint(4, 15), 16, 24, 24, 24, 36, 48, rng.randint(60, 180), 360])
    refine = rng.choice([1, 1, 1, 1, 2, 5, 10]) if entry != "restart" and num_hori <= 48 else 1
    dist = math.exp(rng.uniform(math.log(10e3), math.log(80e3)))
    edge = math.exp(rng.uniform(math.log(0.1), math.log(2.5)))
    most = min(1.5e6, 2.0e7 / (num_hori * refine)) * min(1.0, 40e3 / dist)
    cells = math.exp(rng.uniform(math.log(400.0), math.log(most)))
    n_domains = 1
    if entry == "batch":
        n_domains = rng.randint(2, 20)
        cells = max(400.0, cells / n_domains)
    box = max(math.sqrt(cells * math.sqrt(3.0) / 4.0) * edge, 6.0 * edge)
    hmin = rng.uniform(0.0, 800.0)
    return dict(entry=entry, edge_km=round(edge, 4), box_km=round(box, 3),
                kind=rng.choice(["fbm", "ridged", "eroded"]), hmin=round(hmin, 1),
                hmax=round(hmin + rng.uniform(800.0, 4500.0), 1), num_hori=num_hori,
                grid_type=rng.choice([1, 1, 1, 0]), dist=round(dist, 1),
                ray_org_elev=rng.choice([0.1, 0.2, 0.2, 0.5, 2.0]), refine=refine,
                svf_type=rng.choice([0, 1, 2, 2]),
                precise=rng.random() < 0.15 and entry == "device",
                lat=round(rng.uniform(-65.0, 65.0), 2), lon=round(rng.uniform(-170.0, 170.0), 2),
                rot=round(rng.uniform(0.0, 120.0), 2), n_domains=n_domains)


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

@functools.lru_cache(maxsize=64)
def _grid(lat, lon, box_km, edge_km, rot):
    """A grid's arrays: it stays while the elevations change from seed to seed."""
    return icon_like_grid(lat, lon, box_km, edge_km, rot)


def _domains_of(case):
    """(lat, lon, box_km, edge_km, rot, num_hori) of every domain of a case: the
    domains of a batch differ in size and spacing around the case's values."""
    n = case["n_domains"]
    if n == 1:
        return [(case["lat"], case["lon"], case["box_km"], case["edge_km"], case["rot"],
                 case["num_hori"])]
    out = []
    for k in range(n):
        f = 2.0 ** (1.5 * math.sin(2.4 * k))  # sizes spread over a factor of eight
        edge = case["edge_km"] * (0.6 + 0.8 * ((k * 7) % n) / n)
        box = max(case["box_km"] * edge / case["edge_km"] * math.sqrt(f), 6.0 * edge)
        lat = max(-66.0, min(66.0, case["lat"] + 9.0 * math.sin(1.7 * k)))
        nh = case["num_hori"] if k % 3 else max(4, case["num_hori"] * 2 // 3)
        out.append((lat, case["lon"] + 4.0 * k, box, edge, (case["rot"] + 11.0 * k) % 120.0, nh))
    return out


def _fbm(n, hurst, gen, device):
    """Periodic spectral fractional-Brownian field, n x n, unit deviation."""
    kx = torch.fft.fftfreq(n, device=device, dtype=torch.float64)
    ky = torch.fft.rfftfreq(n, device=device, dtype=torch.float64)
    k = torch.sqrt(kx[:, None] ** 2 + ky[None, :] ** 2)
    amp = torch.where(k > 0, k, torch.ones_like(k)) ** (-(hurst + 1.0))
    amp[0, 0] = 0.0
    re = torch.randn(k.shape, generator=gen, device=device, dtype=torch.float64)
    im = torch.randn(k.shape, generator=gen, device=device, dtype=torch.float64)
    f = torch.fft.irfft2(torch.complex(amp * re, amp * im), s=(n, n))
    f = f - f.mean()
    return f / f.std()


def _sample(f, x, y, extent):
    """Bilinear samples of a periodic field over [-extent / 2, extent / 2]^2."""
    n = f.shape[0]
    u, v = (x / extent + 0.5) * n, (y / extent + 0.5) * n
    i0, j0 = torch.floor(u).long(), torch.floor(v).long()
    fu, fv = u - i0, v - j0
    i0, j0 = i0 % n, j0 % n
    i1, j1 = (i0 + 1) % n, (j0 + 1) % n
    return ((1 - fu) * (1 - fv) * f[j0, i0] + fu * (1 - fv) * f[j0, i1]
            + (1 - fu) * fv * f[j1, i0] + fu * fv * f[j1, i1])


def _unit(h):
    lo, hi = h.min(), h.max()
    return (h - lo) / (hi - lo)


def _elevations(grid, case, box_km, edge_km, seed):
    """Cell elevations [m]: fractional-Brownian terrain, with Gaussian massifs
    (``fbm``) or ridged noise (``ridged``; sharper for ``eroded``)."""
    device = "cuda" if torch.cuda.is_available() else "cpu"
    gen = torch.Generator(device=device)
    gen.manual_seed(seed)
    x = torch.from_numpy(grid["vx"]).to(device)
    y = torch.from_numpy(grid["vy"]).to(device)
    extent = 1250.0 * box_km
    n = int(2 ** min(12, max(8, math.ceil(math.log2(2.5 * box_km / edge_km)))))
    base = _unit(_sample(_fbm(n, 0.7 if case["kind"] == "ridged" else 0.8, gen, device), x, y,
                         extent))
    if case["kind"] == "fbm":
        h = base
        p = torch.rand((12, 4), generator=gen, device=device, dtype=torch.float64).cpu().numpy()
        for cx, cy, sig, amp in p:
            s = 1000.0 * box_km * (0.02 + 0.08 * sig)
            h = h + (0.15 + 0.35 * amp) * torch.exp(
                -((x - (cx - 0.5) * 1000.0 * box_km) ** 2
                  + (y - (cy - 0.5) * 1000.0 * box_km) ** 2) / (2.0 * s * s))
    else:
        g = _sample(_fbm(n, 0.9, gen, device), x, y, extent)
        r = (1.0 - g.abs() / g.abs().max()) ** (2.0 if case["kind"] == "ridged" else 3.0)
        h = 0.55 * base + 0.45 * _unit(r)
    # Small domains keep the slopes of the large ones: the relief over a box
    # grows with its size up to the range named by the case.
    relief = (case["hmax"] - case["hmin"]) * min(1.0, (box_km / 60.0) ** 0.7)
    hv = case["hmin"] + relief * _unit(h)
    voc = torch.from_numpy(grid["vertex_of_cell"].astype(np.int64)).to(device)
    return ((hv[voc[0]] + hv[voc[1]] + hv[voc[2]]) / 3.0).cpu().numpy()


def _inputs(case, seed):
    """[(the six input arrays, num_hori)] of every domain of a case."""
    out = []
    for k, (lat, lon, box, edge, rot, nh) in enumerate(_domains_of(case)):
        g = _grid(lat, lon, box, edge, rot)
        h = _elevations(g, case, box, edge, 1000003 * seed + k)
        out.append(((g["clon"], g["clat"], h, g["vlon"], g["vlat"], g["cells_of_vertex"]), nh))
    return out


def _args(case, num_hori):
    return (num_hori, case["grid_type"], case["dist"], case["ray_org_elev"], case["refine"],
            case["svf_type"])


def prepare(case, seed):
    doms = _inputs(case, seed)
    if case["entry"] == "batch":
        return dict(case=case, domains=[(a, _args(case, nh)) for a, nh in doms])
    arrays, nh = doms[0]
    args = _args(case, nh)
    if case["entry"] == "host":
        return dict(case=case, arrays=arrays, args=args)
    dev = torch.device("cuda", torch.cuda.current_device())
    t = [torch.from_numpy(a).to(dev) for a in arrays]
    nc = t[0].numel()
    state = dict(case=case, arrays=t, args=args,
                 horizon=torch.empty((nh, nc), dtype=torch.float64, device=dev),
                 skyview=torch.empty(nc, dtype=torch.float64, device=dev),
                 options=dict(precision=1) if case["precise"] else {})
    if case["entry"] == "restart":
        # The earlier run: the same grid with the old orography, a few metres
        # off; its horizons in quarter degrees are the start's half degrees.
        raw = torch.empty((nh * case["refine"], nc), dtype=torch.int16, device=dev)
        gen = torch.Generator(device=dev)
        gen.manual_seed(seed + 17)
        old = list(t)
        old[2] = t[2] + 8.0 * torch.randn(nc, generator=gen, device=dev, dtype=torch.float64)
        horizon_svf_comp_device(*old, *args, state["horizon"], state["skyview"], raw_index=raw)
        state["options"] = dict(start_index=torch.div(raw, 2, rounding_mode="floor").contiguous(),
                                mlp_azimuth_groups=-1)
    return state


def run(state):
    case = state["case"]
    if case["entry"] == "batch":
        return horizon_svf_comp_batch(state["domains"])
    if case["entry"] == "host":
        return horizon_svf_comp_py(*state["arrays"], *state["args"])
    horizon, skyview, _ = horizon_svf_comp_device(*state["arrays"], *state["args"],
                                                  state["horizon"], state["skyview"],
                                                  **state["options"])
    return horizon, skyview


def work(case):
    """Inputs once, outputs once; per azimuth of a cell a ray that meets the
    terrain and one that does not, each decided by one triangle."""
    nbytes = flops = 0.0
    for lat, lon, box, edge, rot, nh in _domains_of(case):
        g = _grid(lat, lon, box, edge, rot)
        nc, nv = g["clon"].size, g["vlon"].size
        nbytes += 24.0 * nc + 40.0 * nv + 8.0 * nc * (nh + 1)
        if case["entry"] == "restart":
            nbytes += 2.0 * nc * nh
        flops += 2.0 * 60.0 * nc * nh * case["refine"]
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# The same in 64 bits
# ---------------------------------------------------------------------------

def _triangles(clon, clat, hsurf, vlon, vlat, cov, grid_type):
    """Mesh vertices (lon, lat, h) and triangles: a fan around every ICON vertex
    over its cells in the order of their bearing."""
    valid = cov != -2
    n = valid.sum(axis=0)
    c = np.where(valid, cov, 0)
    ang = np.arctan2(clon[c] - vlon, clat[c] - vlat)
    ang = np.where(ang < 0.0, ang + 2.0 * np.pi, ang)
    order = np.argsort(np.where(valid, ang, np.inf), axis=0, kind="stable")
    c = np.take_along_axis(c, order, axis=0)
    if grid_type == 0:
        tri = [np.stack([c[0], c[k + 1], c[k + 2]], 1)[n >= k + 3] for k in range(4)]
        return clon, clat, hsurf, np.concatenate(tri)
    full = np.nonzero(n == 6)[0]
    ids = clon.size + np.arange(full.size)
    c = c[:, full]
    tri = [np.stack([c[k], c[(k + 1) % 6], ids], 1) for k in range(6)]
    return (np.concatenate([clon, vlon[full]]), np.concatenate([clat, vlat[full]]),
            np.concatenate([hsurf, hsurf[c].mean(axis=0)]), np.concatenate(tri))


def _exact_domain(arrays, num_hori, case):
    clon, clat, hsurf, vlon, vlat, cov = arrays
    device = "cuda" if torch.cuda.is_available() else "cpu"
    lon, lat, h, tri = _triangles(clon, clat, hsurf, vlon, vlat, cov, case["grid_type"])
    r = R_EARTH + h
    xyz = np.stack([r * np.cos(lat) * np.cos(lon), r * np.cos(lat) * np.sin(lon),
                    r * np.sin(lat)], 1)
    nc = clon.size
    q = torch.from_numpy(xyz[:nc]).to(device)
    up = q / q.norm(dim=1, keepdim=True)
    north = torch.tensor([0.0, 0.0, R_EARTH], dtype=torch.float64, device=device) - q
    north = north - (north * up).sum(1, keepdim=True) * up
    north = north / north.norm(dim=1, keepdim=True)
    east = torch.linalg.cross(north, up)
    mid = q.mean(0)  # coordinates relative to the domain's middle
    org = q + up * case["ray_org_elev"] - mid
    t = torch.from_numpy(xyz).to(device)[torch.from_numpy(tri).to(device)] - mid
    v0, e1, e2 = t[:, 0], t[:, 1] - t[:, 0], t[:, 2] - t[:, 0]
    nrm = torch.linalg.cross(e1, e2)
    tfar = float(np.float32(case["dist"]))
    block = max(1, int(4e7) // max(1, tri.shape[0]))

    def hits(cells, d):
        """Whether each ray meets a triangle within reach (Moeller-Trumbore)."""
        out = torch.empty(cells.numel(), dtype=torch.bool, device=device)
        for b in range(0, cells.numel(), block):
            o, w = org[cells[b:b + block]], d[b:b + block]
            # With s = o - v0: det = -w.n, det t = s.n, det u = s.(w x e2),
            # det v = w.(s x e1), expanded into (rays x 3) (3 x triangles).
            det = -(w @ nrm.T)
            dist = o @ nrm.T - (v0 * nrm).sum(1)
            m = torch.linalg.cross(w, o)  # moment of the ray
            u = w @ torch.linalg.cross(v0, e2).T - m @ e2.T
            v = m @ e1.T - w @ torch.linalg.cross(v0, e1).T
            s = torch.sign(det)
            det, u, v, dist = det * s, u * s, v * s, dist * s
            out[b:b + block] = ((det > 0) & (u >= 0) & (v >= 0) & (u + v <= det) & (dist > 0)
                                & (dist <= tfar * det)).any(1)
        return out

    acc = math.radians(0.25)
    refine, L = case["refine"], num_hori * case["refine"]
    shift = 0.0 if refine == 1 else -math.pi / num_hori + math.pi / L
    m = torch.zeros(nc, dtype=torch.long, device=device)  # elevation in half degrees
    horizon = torch.zeros((num_hori, nc), dtype=torch.float64, device=device)
    svf = torch.zeros(nc, dtype=torch.float64, device=device)
    every = torch.arange(nc, device=device)
    for a in range(L):
        th = shift + 2.0 * math.pi * a / L
        flat = math.cos(th) * north + math.sin(th) * east

        def ask(cells):
            e = (2.0 * acc * m[cells])[:, None]
            return hits(cells, torch.cos(e) * flat[cells] + torch.sin(e) * up[cells])

        first = ask(every)
        live = every[first]
        while live.numel():  # upward to the first miss
            m[live] += 1
            live = live[ask(live)]
        live = every[~first]
        live = live[m[live] > -170]
        while live.numel():  # downward to the first hit or the floor
            m[live] -= 1
            live = live[~ask(live)]
            live = live[m[live] > -170]
        hor = torch.clamp((2 * m + torch.where(first, -1, 1)).double() * acc, min=0.0)
        horizon[a // refine] += torch.rad2deg(hor) / refine
        svf += 1.0 - torch.sin(hor) ** (case["svf_type"] + 1)
    return horizon.cpu().numpy(), (svf / L).cpu().numpy()


def exact(case, seed):
    """By brute force over all triangles: for the small domains only."""
    if case["entry"] == "restart":
        return None  # its result depends on the given starts
    pairs = 0.0
    for lat, lon, box, edge, rot, nh in _domains_of(case):
        nc = _grid(lat, lon, box, edge, rot)["clon"].size
        pairs += 12.0 * nc * nc * nh * case["refine"]
    if pairs > 3e10:
        return None
    out = [_exact_domain(a, nh, case) for a, nh in _inputs(case, seed)]
    return out if case["entry"] == "batch" else out[0]
