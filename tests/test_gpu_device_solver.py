"""The eigensolver of the runs that keep their eigenvectors on the device, at the edges of its
plans: test_gpu_tri_resident's sectors through nrg_diagonalization in a child process with
NRG_ENTRY_SOLVER=device (read once per process): by default, without 16-block clusters
(NRG_TRI_CLUSTER=8: on chip up to 384, streamed up to 3496) and on the multi-kernel reduction of
the orders that are too large for either (NRG_TRI_CLUSTER=0)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))

CHILD = """
import sys
sys.path[:0] = [{root!r}, {package!r}, {here!r}]
from nrg_b200 import Context
import test_gpu_tri_resident as t
def factory(inp):
    c = Context(0)
    c.set_model(inp)
    return c
for n in {orders!r}:
    t.test_sector(n, factory)
    print("passed", n)
"""


@pytest.mark.parametrize("env,orders", [
    # on chip: the edges of the plans; streamed: one column, fewer and more columns than updates are
    # kept back, and all numbers of them (7 up to 1407, 6 to 1567, 5 to 1759, 4 to 2015, 3 to 2352, 2
    # to 2832, 1 to 3536); the multi-kernel reduction
    ({}, [129, 159, 160, 161, 255, 256, 257, 319, 320, 321, 383, 384, 385, 511, 512, 513, 545, 640]),
    ({}, [1407, 1500, 1600, 1759, 2100, 2500]),
    ({}, [3300, 3536, 3537]),
    ({"NRG_TRI_CLUSTER": "8"}, [320, 384, 385, 512, 513, 700, 1300]),
    ({"NRG_TRI_CLUSTER": "8"}, [3496, 3497]),
    ({"NRG_TRI_CLUSTER": "0"}, [129, 256, 513]),
])
def test_sectors(env, orders):
    root = os.path.dirname(HERE)
    code = CHILD.format(root=root, package=os.path.join(root, "nrg-mpi_b200"), here=HERE, orders=orders)
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, NRG_ENTRY_SOLVER="device", **env), cwd=root,
                       capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-3000:]
    assert r.stdout.count("passed") == len(orders)
