"""bench.py's result line stays short: a reader of the output's last 16 KB has it whole."""
import json

import bench


def test_tables_go_to_standard_error(capsys):
    line = {"metric": "layers/s", "value": 1.5, "e2e": {"value": 1.0}, "seeds": [{"x": 0.123456789}] * 100,
            "per_gate": [{"gate": "RX", "ms": 1.23456789}] * 700, "trotter": {"energies": [1.0] * 50}}
    bench.report(dict(line))
    out, err = capsys.readouterr()
    got = json.loads(out)
    assert out.count("\n") == 1 and len(out) < 16000
    assert got == {k: v for k, v in line.items() if k not in ("seeds", "per_gate")}
    assert json.loads(err)["details"] == {k: line[k] for k in ("seeds", "per_gate")}
