"""The benchmark's reference arm prints a number of the reference library or none: on a host
where it does not compile, or has not been built, the line says that it is unavailable."""
from __future__ import annotations

import json
import os
import subprocess
import sys

import pytest

from conftest import ROOT

CODE = """
import sys
machine = sys.argv.pop(1)
import bench
bench.platform.machine = lambda: machine
bench.main()
"""
DRIVER = os.path.join(ROOT, "oracle", "_ref", "msbg_ref_driver")


@pytest.mark.parametrize("machine", ["aarch64", "x86_64"])
@pytest.mark.parametrize("workload", ["surface4096", "surface512"])
def test_unavailable_line(machine, workload):
    if machine == "x86_64" and os.path.isfile(DRIVER):
        pytest.skip("the reference library is built here")
    env = {k: v for k, v in os.environ.items() if k not in ("RANK", "WORLD_SIZE", "LOCAL_RANK")}
    out = subprocess.run([sys.executable, "-c", CODE, machine, "--impl", "reference", "--workload", workload, "--steps",
                          "1", "--warmup", "1"], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
    line = json.loads(out.stdout)
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
