"""The autotuner's cache file on the host: choices of an earlier meaning of the fields are not applied."""
import json
from types import SimpleNamespace

import torch


def test_entries_without_the_present_version_are_measured_again(tmp_path, monkeypatch):
    """Up to version 1 sweep_nbuf was a ring depth (2 or 3, always stored): read as the present switch it would
    turn the L2 prefetch off or on regardless of the factors' size."""
    from dac_vtsa_b200 import autotune
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda *_: "NVIDIA B200")
    model = SimpleNamespace(grid=SimpleNamespace(Nr=16, Nth=16, Nz=64), device="cuda:0", n_w=1024,
                            cfg=SimpleNamespace(solver=SimpleNamespace(preconditioner="theta_block")))
    old = {"params": {"sweep_nbuf": 2}, "times_us": {}}
    path = tmp_path / "tune.json"
    path.write_text(json.dumps({"NVIDIA_B200/16x16x64/wall1/theta_block/fp64": old}))
    applied, chosen = [], {"sweep_nbuf": 3}
    monkeypatch.setattr(autotune, "apply", lambda m, p: applied.append(p))
    monkeypatch.setattr(autotune, "tune", lambda m, y, dh: (chosen, {}))
    assert autotune.cached(model, None, 1.0, path=str(path)) == chosen and not applied
    assert autotune.cached(model, None, 1.0, path=str(path)) == chosen and applied == [chosen]
    assert json.loads(path.read_text())["NVIDIA_B200/16x16x64/wall1/theta_block/fp64"] == old
