"""The runner's sweep options choose the sweep that runs, on their own and together."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("args, text", [
    ([], "sweep_exchange=pipelined"),
    (["--sweep-pipeline", "4"], "sweep_cluster=4 sweep_exchange=pipelined"),
    (["--sweep-exchange", "slab"], "sweep_cluster=8 sweep_exchange=slab"),
    (["--sweep-exchange", "shared", "--sweep-cluster", "4"], "sweep_cluster=4 sweep_exchange=shared"),
    (["--sweep-cluster", "2"], "sweep_cluster=2 sweep_exchange=l2")])
def test_sweep_options(args, text):
    p = subprocess.run([sys.executable, "-m", "aerocfd_b200.run", "--case", "bump", "--no-autotune", "--steps", "3",
                        *args], cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stderr
    line = json.loads(p.stdout.strip().splitlines()[-1])
    assert text in line["tuning"] and line["device_status"] == 0
