"""A saved tuning is used by the kernels it was measured on and by no others."""
import json

import pytest

from gs_tmi_b200 import autotune
from gs_tmi_b200._lib import GsvShape

SHAPE = GsvShape(24, 20, 16, 8)


def _keys():
    tuner = autotune.Autotuner
    return tuner.key(SHAPE, 300, False), tuner.key(SHAPE, 300, True), tuner.tile_key((24, 20, 16), 300, False)


def test_picks_without_a_build_are_not_used(tmp_path):
    """The keys that files written before the build was part of them hold."""
    path = tmp_path / "tune.json"
    path.write_text(json.dumps({"24x20x16/ts8/n2^9/atomic": [1, 8], "24x20x16/ts8/n2^9/det": [1, 8],
                                "24x20x16/n2^9/atomic/tile": [4, 2, 32, 1]}))
    assert not set(_keys()) & set(autotune.Autotuner(str(path)).cache)


def test_picks_of_another_build_are_not_used(tmp_path, monkeypatch):
    other = tmp_path / "other.so"
    other.write_bytes(b"another build")
    path = tmp_path / "tune.json"
    path.write_text(json.dumps({k: [2, 16] for k in _keys()}))
    assert set(_keys()) <= set(autotune.Autotuner(str(path)).cache)
    monkeypatch.setattr(autotune, "LIB_PATH", str(other))
    autotune.kernels_id.cache_clear()
    try:
        assert not set(_keys()) & set(autotune.Autotuner(str(path)).cache)
    finally:
        autotune.kernels_id.cache_clear()


@pytest.mark.parametrize("n,bucket", [(0, 0), (1, 0), (300, 9), (512, 9), (513, 10)])
def test_buckets(n, bucket):
    assert f"/n2^{bucket}/" in autotune.Autotuner.key(SHAPE, n, False)
    assert f"/n2^{bucket}/" in autotune.Autotuner.tile_key((24, 20, 16), n, True)
