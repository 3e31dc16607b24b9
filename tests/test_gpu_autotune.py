"""The autotuner with its built-in grid: the profile sweep where it is far ahead of
the tree search, without a descent; the tree search's knobs tuned together where the
sweep's grid cannot hold the domain."""
import numpy as np
import pytest

from horayzon_extpar_gb300 import synthetic

pytestmark = pytest.mark.gpu

ARGS = (24, 1, 20000.0, 0.2, 1, 2)


def _tensors(inputs):
    torch = pytest.importorskip("torch")
    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in inputs]


def test_autotune_keeps_the_sweep_without_a_descent(tmp_path, monkeypatch):
    from horayzon_extpar_gb300 import autotune
    monkeypatch.setenv("HZ_AUTOTUNE_CACHE", str(tmp_path / "tune.json"))
    d = synthetic.make_domain(edge_km=1.0, box_km=60.0, seed=71)
    res = autotune.tune(_tensors(d.inputs()), ARGS)
    assert autotune.knobs(res) == autotune.DEFAULTS and res["trials"] == 2


def test_autotune_descends_from_the_tree_where_the_sweep_cannot_run(tmp_path, monkeypatch):
    from horayzon_extpar_gb300 import autotune
    monkeypatch.setenv("HZ_AUTOTUNE_CACHE", str(tmp_path / "tune.json"))
    a, b = ([np.array(x) for x in
             synthetic.make_domain(edge_km=1.0, box_km=20.0, seed=s).inputs()] for s in (72, 73))
    for k in (0, 3):
        b[k] += 2.0  # 115 degrees further east
    n = a[0].size
    inputs = [np.concatenate([x, y]) for x, y in zip(a[:5], b[:5])]
    inputs.append(np.concatenate([a[5], np.where(b[5] == -2, -2, b[5] + n)], 1))
    res = autotune.tune(_tensors(inputs), ARGS, reps=1, rounds=1)
    assert all(res[k] in v for k, v in autotune.GRID.items())  # a tree setting
    assert res["trials"] == 2 + sum(len(v) - 1 for v in autotune.GRID.values())
