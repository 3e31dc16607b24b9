"""The benchmark's output: one JSON line on stdout that stays short whatever the
extra reports hold, and traffic figures only of the domain they were profiled on."""
import json

import bench


def test_result_line_is_alone_on_stdout_and_short(capsys, tmp_path):
    line = {"metric": "evals/s", "value": 1.0, "reports": ["configs"]}
    reports = {"configs": {"a": list(range(10000))}, "batched_domains": {"b": 2.0}}
    bench.emit(line, reports, str(tmp_path / "r.json"))
    out, err = capsys.readouterr()
    assert out == json.dumps(line) + "\n"
    got = [json.loads(x) for x in err.splitlines()]
    assert [g.pop("report") for g in got] == ["configs", "batched_domains"]
    assert got == list(reports.values())
    assert json.load(open(tmp_path / "r.json")) == {**line, **reports}


def test_traffic_belongs_to_the_profiled_domain():
    _, nbytes, cells = bench.traffic_from_profile(0)
    assert nbytes > 0 and cells == 783073
    assert bench.traffic_from_profile(cells)[0] == nbytes
    assert bench.traffic_from_profile(3141157)[0] is None
