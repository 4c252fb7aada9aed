"""The engines that a context reports are those that it runs, and a tuning file's choice
among the engines of an older library is not taken."""
import json
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]
REPORT = """
import importlib, json, sys
hqt = importlib.import_module("ads4-holographic-quantum-turbulence_b200")
nx, ny, nz, precision, tune = json.loads(sys.argv[1])
with hqt.Simulation(nx, ny, nz, precision=precision, autotune=tune) as sim:
    print(json.dumps(sim.config_report()))
"""


def report(*args, **env):
    """config_report of a context in a process of its own (a tuning file is read once)."""
    out = subprocess.run([sys.executable, "-c", REPORT, json.dumps(args)], cwd=ROOT, check=True,
                         capture_output=True, text=True, env={**os.environ, **env})
    return json.loads(out.stdout.splitlines()[-1])


@pytest.mark.parametrize("precision,engine", [("fp64", "runtime"), ("mixed", "compile-time")])
def test_reported_engine_without_the_prime_factor_one(cuda, precision, engine):
    chosen = report(301, 64, 8, precision, False, HQT_LINE_ENGINE="stockham")["chosen"]
    assert (chosen["x_engine"], chosen["y_engine"]) == (engine, "compile-time")


def test_an_older_librarys_choice_is_tuned_again(cuda, tmp_path):
    f = tmp_path / "tune.txt"
    f.write_text("dev0:64x64x12:fp64:f1:w1 0 0 0 0 1 1 1 1 1\n")
    first = report(64, 64, 12, "fp64", True, HQT_TUNE_CACHE=str(f))
    assert first["cached"] is False
    again = report(64, 64, 12, "fp64", True, HQT_TUNE_CACHE=str(f))
    assert again["cached"] is True and again["chosen"] == first["chosen"]
