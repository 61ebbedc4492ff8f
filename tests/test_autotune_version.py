"""The tuning cache holds choices among one version of the step kernels only."""
import json

import numpy as np
import torch

from hipims_b200 import autotune
from hipims_b200.fused import Catchment


def test_choice_of_other_kernels_is_timed_again(monkeypatch, tmp_path):
    cache = tmp_path / "tune.json"
    monkeypatch.setenv("HIPIMS_B200_TUNE_CACHE", str(cache))
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda device=None: "FakeGPU")
    mask = np.ones((40, 48), np.int32)
    c = Catchment(mask=mask, z=np.zeros(mask.shape), h=np.full(mask.shape, 0.1))
    # an entry as the first version wrote it, and one of the version before this one
    old = {"best": {"tile": [32, 32], "grid_blocks": 0, "minb": 6}, "ms_per_step": 1.0}
    shape = f"FakeGPU|float32|n=1|cells={mask.size}|side=48"
    spinup = f"|spinup={autotune.SPINUP_STEPS}"
    cache.write_text(json.dumps({
        shape + spinup: old,
        f"{shape}|kernels={getattr(autotune, 'KERNELS', 1) - 1}{spinup}": old}))
    timed = []

    def fake_time(cs, dtype, device, cfg, **kw):
        timed.append(cfg)
        return 1.0 if tuple(cfg["tile"]) == (32, 64) and cfg["minb"] == 4 else 2.0

    monkeypatch.setattr(autotune, "time_config", fake_time)
    best = autotune.tune([c], torch.float32, "cpu")
    assert len(timed) == len(autotune.DEFAULT_CANDIDATES)
    assert best["tile"] == (32, 64) and best["minb"] == 4
    timed.clear()
    again = autotune.tune([c], torch.float32, "cpu")
    assert timed == [] and again["tile"] == (32, 64) and again["minb"] == 4
