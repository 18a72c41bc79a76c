"""bench.py prints its one JSON line whatever becomes of the sections after the
headline: one that raises, and one that holds the host in a native call and
does not return."""
import json
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

SCRIPT = """
import ctypes, bench
stuck = lambda: ctypes.CDLL(None).sleep(600)
bench.run_sections({{"metric": "m", "value": 1.5}}, [("a", lambda: 1), ("b", {b}), ("c", lambda: 3)], 2.0, True)
"""


@pytest.mark.parametrize("b,rest", [("lambda: 2", {"b": 2, "c": 3}),
                                    ("lambda: 1 // 0", {"b": {"error": "ZeroDivisionError('integer division or modulo by zero')"},
                                                        "c": 3}),
                                    ("stuck", {"sections_unfinished": "b"})])
def test_the_headline_line_is_printed_once(b, rest):
    r = subprocess.run([sys.executable, "-c", SCRIPT.format(b=b)], capture_output=True, text=True, cwd=ROOT, timeout=60)
    assert r.returncode == 0, r.stderr[-2000:]
    lines = [json.loads(x) for x in r.stdout.splitlines() if x.startswith("{")]
    assert lines == [{"metric": "m", "value": 1.5, "a": 1, **rest}]
