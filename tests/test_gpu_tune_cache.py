"""The autotuner's cache: a plan takes over a cached group size only from plans whose
tasks are alike, and nothing from a file that an earlier scheduler wrote. Each in a
process of its own (the cache is the process's), with a file of its own."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import sys
sys.path.insert(0, %r)
import numpy as np, torch
import pbe_gb300 as pg
torch.zeros(1, device="cuda")
def plan(n, q, cells):
    x = pg.grids.geometric_pow2(n, 1e-21, q)
    with pg.BatchPlan([x], [n] * cells, [0] * cells, 5, tune=True) as p:
        print(p.schedule())
""" % os.path.join(ROOT, "pbe-fixed-pivot-cuda_gb300")


def _run(code, path):
    env = dict(os.environ, PBE_GB300_TUNE_CACHE=str(path))
    out = subprocess.run([sys.executable, "-c", CHILD + code], capture_output=True, text=True, env=env,
                         timeout=300)
    assert out.returncode == 0, out.stderr[-1500:]
    with open(path) as f:
        return f.read().split("\n")[:-1]


def test_plans_of_other_sizes_are_tuned_apart(tmp_path):
    # one class of section counts (128..255): 1 cell and 512 cells; 10 and 176 direct lags
    lines = _run("plan(200, 4.0, 1); plan(200, 4.0, 512); plan(200, 32.0, 512); plan(200, 4.0, 512)",
                 tmp_path / "tune")
    assert len(lines) == len(set(line.rsplit(" ", 1)[0] for line in lines)) == 3, lines


def test_entries_of_earlier_schedulers_are_passed_over(tmp_path):
    path = tmp_path / "tune"
    old = ["%d 5 %d %d 256" % (sms, brk, cls) for sms in (132, 148, 152) for brk in range(4) for cls in range(16)]
    path.write_text("\n".join(old) + "\n")
    lines = _run("plan(200, 4.0, 512)", path)
    assert lines[:len(old)] == old and len(lines) == len(old) + 1, lines[len(old):]


def test_file_is_read_back(tmp_path):
    path = tmp_path / "tune"
    first = _run("plan(200, 4.0, 16); plan(960, 32.0, 4)", path)
    assert len(first) == 2
    assert _run("plan(200, 4.0, 16); plan(960, 32.0, 4)", path) == first
