"""Stored tunings belong to the step kernels that they were timed on."""
import json

import numpy as np


def test_a_file_written_for_other_kernels_is_not_applied(monkeypatch, tmp_path):
    from pysit_gb300 import engine
    rest = (3, 4, (53, 49, 45), str(np.float64), 0, 2, "checkpoint", False, 1)
    path = tmp_path / "tunings.json"
    path.write_text(json.dumps([[repr(rest), 64, [0.0, 0.0, 0.0], 0]]))  # the key before kernels had a name
    monkeypatch.setattr(engine, "_TUNED", {})
    monkeypatch.setattr(engine, "_TUNE_FILES_READ", set())
    monkeypatch.setenv("PYSIT_CUDA_TUNE_CACHE", str(path))
    key = engine._tuning_key(3, 4, [53, np.int64(49), 45], np.float64, 0, 2, "checkpoint", False, 1)
    assert engine._tuning_get(key) is None
    engine._tuning_put(key, (0, (0.0, 0.0, 0.0), 0))
    monkeypatch.setattr(engine, "_TUNED", {})
    monkeypatch.setattr(engine, "_TUNE_FILES_READ", set())
    assert engine._tuning_get(key) == (0, (0.0, 0.0, 0.0), 0)
    assert len(json.loads(path.read_text())) == 2  # the other kernels' tuning stays in the file
