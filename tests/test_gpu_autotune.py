"""The ensemble autotuner times each tile once and serves cached choices only to the
kernels that they were made for."""
import json

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,expect", [("fp64", {32: [0], 64: [0, 1], 128: [0, 1], 256: [0, 1, 2], 512: [0, 2]}),
                                              ("fp32", {32: [0], 64: [0, 1, 2], 128: [0, 1, 2], 256: [0, 1, 2], 512: [0, 1, 2]})])
def test_each_tile_is_timed_once(dd, cuda, tmp_path, monkeypatch, precision, expect):
    ens = dd.ensemble.BoussinesqEnsemble2D([32] * 2 + [64] * 2 + [128] * 2 + [256] * 2 + [512], precision=precision)
    tried = {c.n: [] for c in ens.classes}

    def timed(dt, reps=3):
        for c in ens.classes:
            if c.ysched not in tried[c.n]:
                tried[c.n].append(c.ysched)
        return 1.0
    monkeypatch.setattr(ens, "_time_schedule", timed)
    ens.autotune(1e-2, cache=str(tmp_path / "tune.json"))
    assert tried == expect


def test_schedules_of_other_kernels_are_not_served(dd, cuda, tmp_path, monkeypatch):
    """An entry under the key without a revision, or with another one, is left alone."""
    import torch
    cache = tmp_path / "tune.json"
    stale = {"chunks": [1, 1], "ysched": [0, 1], "order": [0, 1], "ms_per_step": 1.0, "when": ""}
    key = "%s|fp64|32,64|2,2" % torch.cuda.get_device_name(cuda)
    db = {key: stale, key + "|r%d" % (dd.ensemble.SCHEDULE_REV - 1): stale}
    cache.write_text(json.dumps(db))

    def tuned():
        ens = dd.ensemble.BoussinesqEnsemble2D([32] * 2 + [64] * 2)
        monkeypatch.setattr(ens, "_time_schedule", lambda dt, reps=3: 1.0)     # nothing is faster than the defaults
        ens.autotune(1e-2, cache=str(cache))
        return [c.chunk for c in ens.classes], [c.ysched for c in ens.classes]
    assert tuned() == ([2, 2], [0, 0])
    after = json.loads(cache.read_text())
    assert len(after) == 3 and all(after[k] == stale for k in db)
    mine = next(k for k in after if k not in db)
    after[mine] = dict(stale, chunks=[2, 1])
    cache.write_text(json.dumps(after))
    assert tuned() == ([2, 1], [0, 1])
