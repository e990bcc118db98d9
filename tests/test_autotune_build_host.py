"""Tile tables belong to the build of the library they were measured on (no
GPU: the measurement is a stand-in)."""
import json

from exocubed_b200 import _native as nat
from exocubed_b200 import autotune
from exocubed_b200 import workloads as W

CFG = W.dry_atmosphere_config(N=24, L=32, precision=1)
K = nat.EXO_K_IMPLICIT


def test_another_builds_table_is_measured_anew(tmp_path, monkeypatch):
    path = str(tmp_path / "tiles.json")
    # what an earlier version of the package left
    with open(path, "w") as f:
        json.dump({autotune.config_key(CFG): {str(K): {"32": 1.0, "64": 2.0}}}, f)
    calls = []

    def measure(cfg):
        calls.append(cfg)
        return {K: {32: 4.0, 64: 3.0}}

    monkeypatch.setattr(autotune, "measure", measure)
    monkeypatch.setattr(autotune, "build_id", lambda: "a")
    assert autotune.best_tiles(CFG, autotune.TileCache(path))[K] == 64 and len(calls) == 1
    assert autotune.best_tiles(CFG, autotune.TileCache(path))[K] == 64 and len(calls) == 1
    monkeypatch.setattr(autotune, "build_id", lambda: "b")
    autotune.best_tiles(CFG, autotune.TileCache(path))
    assert len(calls) == 2
    # the earlier version still finds its own
    assert autotune.TileCache(path).tables[autotune.config_key(CFG)] == {K: {32: 1.0, 64: 2.0}}


def test_build_id_follows_the_file(tmp_path):
    ids = []
    for n, text in enumerate((b"one", b"two", b"one")):
        p = tmp_path / f"lib{n}.so"
        p.write_bytes(text)
        ids.append(autotune.build_id(str(p)))
    assert ids[0] == ids[2] != ids[1]
