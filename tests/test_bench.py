"""The benchmark's host side: what must not cost the headline line, and what the reference arm loads."""

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
