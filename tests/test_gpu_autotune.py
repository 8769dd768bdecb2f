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
