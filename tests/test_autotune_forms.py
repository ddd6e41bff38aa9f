"""The autotuner's candidates include the forms that calls take by default, and its cache is read
for the library version it was written with."""
import json

import numpy as np
import pytest

from npbench_gb300 import _lib, autotune


def test_default_forms_are_candidates():
    jacobi = autotune._space("jacobi_2d", np.float64)
    limbs = [c for c in jacobi if c["JACOBI_HW_WARPS"] == -1 and c["JACOBI_BANDS"] == 0 and "JACOBI_TMA" not in c]
    assert len({c["JACOBI_CHUNK"] for c in limbs}) >= 5 and {c["JACOBI_CHUNK"] for c in limbs} >= {0, 2, 6, 16}
    for dtype in (np.float64, np.float32):
        rows = [c for c in autotune._space("heat_3d", dtype) if c["HEAT_ROWS"] == 0]
        assert {c["HEAT_CHUNK"] for c in rows} >= {0, 1, 2, 4}
        assert all(c["HEAT_HW_ROWS"] == -1 for c in rows)


def test_entries_of_another_version_are_passed_over(tmp_path, monkeypatch):
    shipped = tmp_path / "shipped.json"
    shipped.write_text(json.dumps({"heat_3d/float64/c5x5x5": {"config": {"HEAT_CHUNK": 2}, "library": "any"}}))
    monkeypatch.setattr(autotune, "SHIPPED_PATH", str(shipped))
    monkeypatch.setenv("NPBGB_TUNE_CACHE", str(tmp_path / "tune.json"))
    entry = {"config": {"HEAT_ROWS": 1, "HEAT_HW_ROWS": 3}}
    try:
        for library, want in (("npbgb 0.1.0 sm_103a", {"HEAT_CHUNK": 2}), (_lib.version(), entry["config"]),
                              (None, entry["config"])):
            cached = dict(entry, library=library) if library else entry
            (tmp_path / "tune.json").write_text(json.dumps({"heat_3d/float64/c5x5x5": cached}))
            autotune.load_cache(refresh=True)
            assert autotune.lookup("heat_3d/float64/c5x5x5")["config"] == want
    finally:
        monkeypatch.undo()
        autotune.load_cache(refresh=True)


@pytest.mark.gpu
@pytest.mark.parametrize("bench, shape", [("jacobi_2d", (40, 70)), ("heat_3d", (9, 11, 34))])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_every_candidate_leaves_the_same_bits(bench, shape, dtype):
    pytest.importorskip("torch")
    entry = autotune.tune(bench, shape, dtype, tsteps=3, repeats=1, store=False)
    assert entry["candidates"] == len(autotune._space(bench, dtype)) and entry["ms"] <= entry["default_ms"]
