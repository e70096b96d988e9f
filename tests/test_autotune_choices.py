"""Which cluster sizes the autotuner times and keeps (CPU, with made-up times): the correlation kernel's own choice is
timed where it is one, and stands unless another is clearly faster; a result tuned for another kernel is not taken."""
import json
from types import SimpleNamespace

import pytest

from gisapr_gb300 import _native as nat
from gisapr_gb300.autotune import Autotuner


def _tuner(monkeypatch, path, times, box=128, crop=12, psi=3):
    """A tuner whose correlation takes times[cluster] milliseconds, a job of that shape, and what was set."""
    import torch
    set_to = {}
    real = nat.call

    def call(name, *args):
        if name == "gisapr_set_tuning":
            set_to[args[1]] = args[3]
        else:
            real(name, *args)

    monkeypatch.setattr(nat, "call", call)
    monkeypatch.setattr(nat.Context, "for_device", classmethod(lambda cls, dev: SimpleNamespace(handle=None)))
    monkeypatch.setattr(nat, "DEFAULT_TUNING", {})
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda dev: "GPU")
    monkeypatch.setattr(Autotuner, "_time_correlate", lambda self, *a, **k: times[set_to[nat.TUNE_CORR_CLUSTER]])
    monkeypatch.setattr(Autotuner, "_time_templates", lambda self, *a, **k: 1.0)
    job = SimpleNamespace(device="cuda:0", records=[None] * 5000, cfg=SimpleNamespace(new_box=box, crop=crop), n_psi=psi)
    return Autotuner(path), job


@pytest.mark.parametrize("box, crop, psi", [(64, 10, 3), (128, 12, 3), (192, 12, 3), (256, 14, 3), (256, 14, 40)])
def test_the_kernels_own_choice_stands(native_lib, monkeypatch, tmp_path, box, crop, psi):
    times = {k: 1.0 + 0.1 * k for k in range(9)}
    times[4] = 0.99  # within what two runs differ by
    tuner, job = _tuner(monkeypatch, tmp_path / "t.json", times, box, crop, psi)
    r = tuner.tune(job, n_cand=8, precision="fp32")
    assert r.corr_cluster == 0
    assert {k for k in r.times_ms if "cluster" in k} == {f"plain_cluster_{k}" for k in (0, 1, 2, 3, 4, 5, 6, 8)}
    assert nat.DEFAULT_TUNING[(nat.TUNE_CORR_CLUSTER, box)] == 0


def test_a_clearly_faster_number_is_taken(native_lib, monkeypatch, tmp_path):
    times = {k: 1.0 for k in range(9)}
    times.update({2: 0.9, 3: 0.8995, 5: 0.95})
    tuner, job = _tuner(monkeypatch, tmp_path / "t.json", times)
    assert tuner.tune(job, n_cand=8, precision="fp32").corr_cluster == 3


def test_the_general_kernels_default_is_one_of_the_others(native_lib, monkeypatch, tmp_path):
    times = {k: 1.0 / k for k in range(1, 9)}
    tuner, job = _tuner(monkeypatch, tmp_path / "t.json", times, box=32, crop=6)
    r = tuner.tune(job, n_cand=8, precision="fp32")
    assert r.corr_cluster == 8 and "plain_cluster_0" not in r.times_ms


def test_a_result_of_another_kernel_is_not_taken(native_lib, monkeypatch, tmp_path):
    path = tmp_path / "t.json"
    tuner, job = _tuner(monkeypatch, path, {k: 1.0 + k for k in range(9)})
    old = dict(key="old", size=128, corr_cluster=5, tc_chunk=8)
    path.write_text(json.dumps({f"GPU|n=128|crop=12|psi=3|particles~4096|cand=8|{p}": old for p in ("fp32", "fp16x3")}))
    assert tuner.tune(job, n_cand=8, precision="fp32").corr_cluster == 0
    kept = json.loads(path.read_text())
    assert len(kept) == 3  # the old ones, untouched, and this one
    again = tuner.tune(job, n_cand=8, precision="fp32")  # from the file
    assert again.corr_cluster == 0 and len(json.loads(path.read_text())) == 3
