"""CPU test of the benchmark's reference arm: its rate is that of one step, whatever the number of steps it timed."""
import argparse
import json

import pytest

import bench
from megamol_gb300 import synth


@pytest.mark.parametrize("steps", [1, 4])
def test_rate_of_a_step(monkeypatch, capsys, steps):
    f = synth.uniform(n=1000, edge=10.0, res=16, seed=1)
    monkeypatch.setattr(bench, "make_workload", lambda name: (f, {"workload": name, "kernel": "bump sigma=1"}))
    monkeypatch.setattr(bench, "density_params", lambda desc: {"kernel": 0})
    monkeypatch.setattr(bench, "cpu_pipeline", lambda *a: dict(
        value=1.0, kind="port", s_density=0.5, s_mip=0.25, s_ao=0.125, particles=f.n, ao_particles=250, s_step=0.875))
    bench.run_reference(argparse.Namespace(workload="mixed_phase_64M", warmup=0, steps=steps, gpus=1))
    line = json.loads(capsys.readouterr().out)
    assert line["value"] == pytest.approx(1.0 / (0.5 / 1000 + 0.25 / 1000 + 0.125 / 250), rel=1e-12)
    assert line["value"] == line["cpu_baseline"]["value"] == line["e2e"]["value"]
    assert line["ms_per_step"] == pytest.approx(875.0) and line["steps"] == steps
    assert line["stages_s_per_step"] == {"s_density": 0.5, "s_mip": 0.25, "s_ao": 0.125}
