"""The autotuner's cache holds what was measured: another limiter, or the winds switched off, is another
problem.  No GPU (the fake instance of test_autotune_host)."""
import pytest

pytest.importorskip("torch")
autotune = pytest.importorskip("nebulaviewer_gb300.autotune")
from test_autotune_host import FakeSim  # noqa: E402


def test_limiter_and_winds_are_part_of_the_key(monkeypatch):
    monkeypatch.setattr(autotune, "_CACHE", {})
    keys = set()
    for limiter in ("minmod", "vanleer"):
        for wind in (0.0, 0.5):
            s = FakeSim()
            s.P = dict(s.P, limiter=limiter, wind=wind)
            keys.add(autotune._key(s))
            autotune.autotune(s, knobs=["chunk_i"])
    assert len(keys) == 4 and set(autotune._CACHE) == keys
