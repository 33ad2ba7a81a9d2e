"""bench.py's result is one short JSON line on stdout (no GPU); the records of the
other workloads, many times its size, go to stderr."""
import json

import bench


def test_one_short_line(capsys):
    big = {"serving": {"rows": [{"x": i, "text": "y" * 40} for i in range(400)]}}
    bench.emit({"metric": bench.METRIC, "value": 0.5, "configs": big, "clocks": {"sm_mhz": 2070.0}})
    out, err = capsys.readouterr()
    assert out.count("\n") == 1 and len(out) < 4096
    assert json.loads(out) == {"metric": bench.METRIC, "value": 0.5, "clocks": {"sm_mhz": 2070.0}}
    assert json.loads(err) == {"configs": big}


def test_without_other_workloads(capsys):
    bench.emit({"value": 1.0})
    out, err = capsys.readouterr()
    assert json.loads(out) == {"value": 1.0} and err == ""
