"""The benchmark where the reference's compiled kernels are not built: its
reference arm says so and ends well, and its own arm takes the oracle's
table-driven kernels for the CPU sample."""

import argparse
import json

import numpy as np

import bench
from pelephysics_b200 import workloads


def test_reference_arm_says_that_it_is_unavailable(oracle, monkeypatch, capsys):
    monkeypatch.setattr(oracle, "have_ref", lambda mech: False)
    assert bench.reference_arm(argparse.Namespace(steps=1, warmup=1, gpus=1)) == 0
    lines = capsys.readouterr().out.strip().splitlines()
    assert len(lines) == 1
    line = json.loads(lines[0])
    assert set(line) == {"impl", "unavailable"} and line["impl"] == "reference"


def test_cpu_sample_without_the_reference_kernels(oracle, monkeypatch):
    monkeypatch.setattr(oracle, "have_ref", lambda mech: False)
    eos, species, mw = bench.oracle_eos(oracle, bench.MECH)
    cells = workloads.drm19_field(4, eos=eos, species=species, mw=mw)
    secs, rY, flag, stats = bench.run_cpu(oracle, cells, np.arange(4))
    assert flag == 0 and secs > 0 and np.all(np.isfinite(rY)) and np.all(stats[:, 0] > 0)
