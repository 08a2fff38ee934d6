"""The benchmark's host side: what must not cost the headline line, and what the reference arm loads."""

import json
import subprocess
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
sys.path.insert(0, str(ROOT))


def test_an_error_in_a_side_record_is_recorded():
    import bench

    from fastddm_gb300._lib import FddmError

    def fails(code, message):
        raise FddmError(code, message)

    assert bench.side_record(fails, 4, "does not fit") == {"error": "FddmError: fddm_b200 error 4: does not fit"}
    assert bench.side_record(lambda a: a, {"p50_ms": 1.0}) == {"p50_ms": 1.0}


def test_the_serving_record_is_guarded():
    """run_ours reaches the serving replay only through side_record."""
    src = (ROOT / "bench.py").read_text()
    body = src[src.index("def run_ours"):src.index("def run_validate")]
    assert "side_record(serve_records," in body and "serve_records(args" not in body


def test_the_reference_arm_loads_nothing_of_the_package():
    child = """
import json, sys
sys.argv = ["bench.py", "--impl", "reference", "--config", "small", "--steps", "1", "--warmup", "0"]
import bench
if __name__ == "__main__":
    bench.main()
    maps = open("/proc/self/maps").read()
    print(json.dumps([m for m in sys.modules if m.startswith("fastddm")] + ["library"] * ("libfddm" in maps)))
"""
    r = subprocess.run([sys.executable, "-c", child], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    line, loaded = r.stdout.strip().splitlines()[-2:]
    assert json.loads(line)["impl"] == "reference" and json.loads(loaded) == []
