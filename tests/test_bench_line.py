"""The bench's headline line stays short enough for a log to keep it whole: the other
workloads' rows are not part of it."""
import ast
import os

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_headline_line_carries_no_extra_rows():
    tree = ast.parse(open(os.path.join(REPO, "bench.py")).read())
    run = next(f for f in tree.body if isinstance(f, ast.FunctionDef) and f.name == "run_ours")
    line = next(a.value for a in ast.walk(run) if isinstance(a, ast.Assign) and isinstance(a.value, ast.Dict)
                and getattr(a.targets[0], "id", "") == "line")
    keys = {k.value for k in line.keys}
    assert {"metric", "value", "unit", "ms_per_step", "e2e", "gpu_launches", "clocks", "config"} <= keys
    assert not keys & {"extra", "summary"}
    prints = [c for c in ast.walk(run) if isinstance(c, ast.Call) and getattr(c.func, "id", "") == "print"
              and not any(k.arg == "file" for k in c.keywords)]
    assert len(prints) == 1                      # one line on stdout
