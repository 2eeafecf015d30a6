"""Device memory of the simulations: two 32-bit numbers a neighbour and node (the
neighbour's cell, its rank), at most 72 bytes a node and category beside them (grid
arrays, paths, levels, draws), and 256 MB of weights, each buffer with its eighth of
room. A third number a neighbour, or weights of all nodes at once, exceeds the sum.

The engine's buffers stay with the process, so each call runs in one of its own."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
SCRIPT = r"""
import sys
sys.path[:0] = [%r, %r]
import conftest
import numpy as np
import torch
import helpers as H
from geo_bsd import workloads as WL

def run(dims, kind, k):
    n = dims[0] * dims[1] * dims[2]
    rng = np.random.default_rng(1)
    idx = rng.choice(n, n // 100, replace=False)
    mask = np.zeros(n, np.uint8)
    mask[idx] = 1
    cov = WL.CovSpec(WL.EXPONENTIAL, (9.0, 9.0, 6.0), (0.0, 0.0, 0.0), 1.0, 0.05)
    if kind == "sgs":
        data = np.zeros(n, np.float32)
        data[idx] = rng.standard_normal(len(idx)).astype(np.float32)
        H.engine_sgs(dims, data, mask, cov, (9, 9, 6), k, 3)
    else:
        data = np.zeros(n, np.uint8)
        data[idx] = rng.integers(0, 3, len(idx))
        H.engine_sis(dims, data, mask, [cov] * 3, [(9, 9, 6)] * 3, [k] * 3, [0.5, 0.3, 0.2], 3)

kind, k = sys.argv[1], int(sys.argv[2])
run((12, 11, 10), kind, k)  # the context and the kernels
free = torch.cuda.mem_get_info()[0]
dims = (150, 100, 80)
run(dims, kind, k)
n, systems = dims[0] * dims[1] * dims[2], 1 if kind == "sgs" else 3
taken, most = free - torch.cuda.mem_get_info()[0], 1.125 * (n * systems * (8 * k + 72) + (256 << 20)) + (32 << 20)
print(taken / 1e6, most / 1e6)
assert taken <= most
"""


@pytest.mark.parametrize("kind,k", [("sgs", 32), ("sis", 24)])
def test_two_numbers_a_neighbour(kind, k):
    done = subprocess.run([sys.executable, "-c", SCRIPT % (HERE, os.path.join(HERE, "..", "hpgl-reborn_b200")), kind,
                           str(k)], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stdout + done.stderr
