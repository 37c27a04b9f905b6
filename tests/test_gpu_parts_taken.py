"""A single solve does form its Q-matrix parts at the same time, and does not fall back
to forming them in turn: counted by the phase timers (QED_PROFILE) of a process of its
own."""
import os
import re
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import numpy as np, pyqcm_b200 as qed
from pyqcm_b200 import workloads as W
from tests.helpers import c2v_golden, c2v_problem
rng = np.random.default_rng(4)
for i, p in enumerate([W.plaquette_bath(rng.uniform(-2, 2, 8), rng.uniform(0.1, 1, 8), U=6.0),
                       W.hubbard_cluster(3, 2, U=5.0, mu=2.2, M=0.3), c2v_problem(c2v_golden(), True)]):
    qed.load_problem(p, 1 + i, model_name=f"taken{i}")
    qed.Green_function_solve(1 + i)
"""


def test_parts_run_at_the_same_time():
    r = subprocess.run([sys.executable, "-c", PROGRAM], capture_output=True, text=True, cwd=ROOT, timeout=300,
                       env=dict(os.environ, QED_PROFILE="1"))
    assert r.returncode == 0, r.stderr
    m = re.search(r"Q-matrix parts at the same time\s+\S+ s\s+(\d+) calls", r.stderr)
    assert m and int(m[1]) == 3, r.stderr
