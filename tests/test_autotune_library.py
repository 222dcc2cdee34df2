"""Cached launch shapes are those of the library that was timed: another library's, or one timed before
the library's contents were part of the key, count as missing (an explicit tile from kernels that
have changed since would keep a small mesh from the resident kernel)."""
import json

import cfd_optimisations_b200 as H
from cfd_optimisations_b200 import autotune as A

TILE_64 = dict(kernel=H.KERNEL_TILED, tile=64, tile2=0, block=64, ms_per_step=0.01)


def _libraries(tmp_path):
    paths = []
    for name, data in (("a", b"kernels"), ("b", b"other kernels")):
        p = tmp_path / f"lib{name}.so"
        p.write_bytes(data)
        paths.append(str(p))
    return paths


def test_a_winner_belongs_to_its_library(tmp_path, monkeypatch):
    cache = tmp_path / "autotune.json"
    monkeypatch.setenv("HCFD_AUTOTUNE_CACHE", str(cache))
    monkeypatch.setattr(A, "gpu_name", lambda: "B200")
    a, b = _libraries(tmp_path)
    monkeypatch.setattr(A.native, "LIB_PATH", a)
    cache.write_text(json.dumps({A._key("solver", 15, H.FP64, H.LIMITER_BJ): {"best": TILE_64},
                                 A._key("arena", 15, H.FP32, H.LIMITER_BJ): {"best": dict(tile=64)}}))
    assert A.best_solver_shape(25_600, tune=False)["tile"] == 64
    assert A.best_arena_tile(25_600, H.FP32, tune=False) == 64
    monkeypatch.setattr(A.native, "LIB_PATH", b)
    assert A.best_solver_shape(25_600, tune=False) == A.DEFAULT_SHAPE
    assert A.best_arena_tile(25_600, H.FP32, tune=False) == 128


def test_winners_without_a_library_count_as_missing(tmp_path, monkeypatch):
    cache = tmp_path / "autotune.json"
    monkeypatch.setenv("HCFD_AUTOTUNE_CACHE", str(cache))
    monkeypatch.setattr(A, "gpu_name", lambda: "B200")
    cache.write_text(json.dumps({"B200|solver|fp64|lim0|c15": {"best": TILE_64}}))
    assert A.best_solver_shape(25_600, tune=False) == A.DEFAULT_SHAPE


def test_without_a_library_the_default_shape(tmp_path, monkeypatch):
    monkeypatch.setenv("HCFD_AUTOTUNE_CACHE", str(tmp_path / "autotune.json"))
    monkeypatch.setattr(A, "gpu_name", lambda: "B200")
    monkeypatch.setattr(A.native, "LIB_PATH", str(tmp_path / "not_built.so"))
    assert A.best_solver_shape(25_600, tune=False) == A.DEFAULT_SHAPE
    assert A.best_arena_tile(25_600, H.FP32, tune=False) == 128
