"""The checked build (-DHZ_CHECKED=1) on the profile sweep: its triangles, lists,
grid cells, elevations, queue slots, work positions, result slots and error bounds
are checked on the device, and parity cases run clean through it: runs of several
azimuths, holes in the mesh (repair by rays), refined azimuths, the local-precision
mode, given starts, a batch. The tree search's own checks run on the precise frame
and a batch too, which name a tree option for it."""
import os
import re
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = textwrap.dedent("""
    import sys
    import numpy as np
    import torch
    from horayzon_extpar_gb300 import (horizon_svf_comp_device, horizon_svf_comp_py, synthetic)
    from horayzon_extpar_gb300.horizon_svf import horizon_svf_comp_batch

    def step(name):
        sys.stdout.flush()
        sys.stderr.write("case %s\\n" % name)
        sys.stderr.flush()

    def same(name, inputs, args, **kw):
        step(name + " tree")
        h0, s0, st0 = horizon_svf_comp_py(*inputs, *args, return_stats=True, leaf_size=2, **kw)
        step(name + " sweep")
        h1, s1, st1 = horizon_svf_comp_py(*inputs, *args, return_stats=True, **kw)
        assert st1["search"] == "sweep" and st0["search"] == "tree"
        assert np.array_equal(h0, h1) and np.array_equal(s0, s1)
        assert st0["num_rays"] == st1["num_rays"]

    d = synthetic.make_domain(edge_km=2.5, box_km=60.0, seed=21)
    same("plain", d.inputs(), (24, 1, 40000.0, 0.2, 1, 2))
    d = synthetic.make_domain(edge_km=0.5, box_km=95.0, seed=10, hmax=3000.0)
    same("runs", d.inputs(), (77, 1, 6000.0, 0.2, 1, 2))
    d = synthetic.make_domain(edge_km=0.5, box_km=30.0, seed=12)
    clon, clat, h, vlon, vlat, cov = (np.array(a) for a in d.inputs())
    cov[:, np.random.default_rng(12).random(cov.shape[1]) < 0.1] = -2
    same("holes", (clon, clat, h, vlon, vlat, cov), (24, 0, 20000.0, 0.2, 3, 0))
    d = synthetic.make_domain(edge_km=0.2, box_km=8.0, seed=15, kind="eroded", hmax=3000.0)
    same("precise", d.inputs(), (60, 1, 8000.0, 0.2, 1, 2), precision=1)
    # Rays far along the diagonals of the domain's axes, and origins far above flat
    # terrain: where a bound by horizontal distance alone falls short.
    d = synthetic.make_domain(edge_km=10.0, box_km=1200.0, seed=16, hmax=9000.0)
    same("far", d.inputs(), (8, 1, 500000.0, 0.2, 1, 2))
    d = synthetic.make_domain(edge_km=0.5, box_km=20.0, seed=7, hmin=100.0, hmax=100.0,
                              n_features=0)
    same("above", d.inputs(), (8, 1, 40000.0, 2000.0, 1, 2))
    d = synthetic.make_domain(edge_km=0.2, box_km=8.0, seed=15, kind="eroded", hmax=3000.0)
    step("starts sweep")
    t = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in d.inputs()]
    g = torch.Generator().manual_seed(5)
    start = torch.randint(-200, 200, (24, d.ncell), generator=g).to(torch.int16).cuda()
    horizon_svf_comp_device(*t, 24, 1, 8000.0, 0.2, 1, 2, start_index=start,
                            mlp_azimuth_groups=4)
    batch = [(d.inputs(), a) for d, a in
             synthetic.make_batch(n_domains=4, seed=3, min_cells=300, max_cells=3000)]
    step("batch tree")
    a = horizon_svf_comp_batch(batch, leaf_size=2)
    step("batch sweep")
    b = horizon_svf_comp_batch(batch)
    assert all(np.array_equal(x[0], y[0]) and np.array_equal(x[1], y[1]) for x, y in zip(a, b))
    step("end")
    print("checked build: clean")
""")

# Bits of hz_ray.cuh's kCheck*.
NODE, LEAF, OUTPUT, TRIANGLE, LIST, GRID, ELEVATION, QUEUE, POSITION, SLOT, BOUND = (
    1 << k for k in range(1, 12))
SWEEP = BOUND | TRIANGLE | LIST | GRID | ELEVATION | QUEUE | POSITION | SLOT | OUTPUT


def test_gpu_checked_build_checks_the_sweep(tmp_path):
    from horayzon_extpar_gb300 import _build
    lib = _build.build_checked(str(tmp_path / "checked"))
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, HZ_LIBRARY=lib,
               PYTHONPATH=root + os.pathsep + os.environ.get("PYTHONPATH", ""))
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=root, env=env,
                       capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "checked build: clean" in r.stdout
    made = {}
    for part in r.stderr.split("case ")[1:]:
        made[part.split("\n", 1)[0]] = [int(m, 16) for m in
                                        re.findall(r"^hz_checks ([0-9a-f]+)$", part, re.M)]
    assert len(made) == 16 and made.pop("end") == []
    for name, masks in made.items():
        want = SWEEP if name.endswith("sweep") else NODE | LEAF
        assert masks and all(m & want == want for m in masks), (name, masks)
