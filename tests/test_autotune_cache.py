"""The autotuner's cache (CPU): tuned values are stored per device under
$XDG_CACHE_HOME and read back by a fresh process state, including the
checkpoint interval k of gauge runs and the per-arithmetic tile heights."""
import json

from diffswe2d_b200 import autotune


def test_cache_round_trip(tmp_path, monkeypatch):
    monkeypatch.setenv("XDG_CACHE_HOME", str(tmp_path))
    monkeypatch.setattr(autotune, "_device_key", lambda device: "TestGPU/148")
    monkeypatch.setattr(autotune, "_tuned", {})
    entry = autotune._load("cuda")
    assert entry == {}
    entry["rows"] = [8, 16, 32, 8]
    entry["rows_fast"] = [16, 16, 32, 16]
    entry["checkpoint_every"] = {
        "exact/4x244x393/1125x0.02/6g/auto": {"k": 64, "timing_ms": {"32": 9.0, "64": 7.5},
                                               "intervals_timed": 300}}
    autotune._store("cuda", entry)
    on_disk = json.loads((tmp_path / "diffswe2d_b200" / "autotune.json").read_text())
    assert on_disk["TestGPU/148"]["checkpoint_every"]["exact/4x244x393/1125x0.02/6g/auto"]["k"] == 64
    monkeypatch.setattr(autotune, "_tuned", {})  # a new process
    assert autotune.tuned_rows(5000, "cuda") == 8
    assert autotune.tuned_rows(5000, "cuda", "fast") == 16
    assert autotune.tuned_rows(1 << 24, "cuda", "fast") == 16
    got = autotune.checkpoint_tuning("cuda", "exact/4x244x393")
    assert list(got.values())[0]["k"] == 64


def test_defaults_without_cache(tmp_path, monkeypatch):
    monkeypatch.setenv("XDG_CACHE_HOME", str(tmp_path))
    monkeypatch.setattr(autotune, "_device_key", lambda device: "Other/1")
    monkeypatch.setattr(autotune, "_tuned", {})
    assert autotune.tuned_rows(100, "cuda") == autotune.DEFAULT_ROWS[0]
    assert autotune.tuned_ensemble_rows("cuda", "fast") == 16
    assert autotune.checkpoint_tuning("cuda") == {}


def test_heights_are_timed_only_where_steps_are_swept(tmp_path, monkeypatch):
    """IEEE grids that take shared-memory tiles have no height: nothing is
    timed or stored for them."""
    monkeypatch.setenv("XDG_CACHE_HOME", str(tmp_path))
    monkeypatch.setattr(autotune, "_device_key", lambda device: "TestGPU/148")
    monkeypatch.setattr(autotune, "_tuned", {})
    timed = []
    monkeypatch.setattr(autotune, "_time_steps",
                        lambda ny, nx, r, *a, **k: timed.append((ny, nx, r)) or 1.0 + abs(r - 32))
    assert autotune.tuned_rows_for_shape(1, 244, 393) == 0 and not timed
    assert autotune._load("cuda").get("shapes", {}) == {}
    assert autotune.tuned_rows_for_shape(1, 244, 393, arithmetic="fast") == 32
    assert [r for _, _, r in timed] == list(autotune.ROW_CHOICES)
    timed.clear()
    assert autotune.tuned_rows_for_shape(17, 244, 393) == 32 and timed  # 1.63 million cells
    timed.clear()
    monkeypatch.setattr(autotune, "_tune_chunk", lambda device: 32)
    monkeypatch.setattr(autotune, "_tune_ensemble_rows", lambda device, arithmetic: 16)
    assert autotune.tune()["rows"] == [0, 0, 0, 32]
    assert {(ny, nx) for ny, nx, _ in timed} == {(2048, 2048)}
