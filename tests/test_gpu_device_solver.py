"""The eigensolver of the runs that keep their eigenvectors on the device, at the edges of its
plans: test_gpu_tri_resident's sectors through nrg_diagonalization in a child process with
NRG_ENTRY_SOLVER=device (read once per process), by default and on the multi-kernel reduction
of the orders that are too large for it (NRG_TRI_CLUSTER=0)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def run_child(env, args, passed):
    cmd = [sys.executable, "-m", "pytest", "-q", "-x", "-p", "no:cacheprovider"] + args
    r = subprocess.run(cmd, env=dict(os.environ, NRG_ENTRY_SOLVER="device", **env), cwd=os.path.dirname(HERE),
                       capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-3000:]
    assert f"{passed} passed" in r.stdout


@pytest.mark.parametrize("env,orders", [
    ({}, [129, 159, 160, 161, 255, 256, 257, 319, 320, 321, 383, 384, 385, 511, 512, 513, 545, 640, 1500, 2100]),
    ({"NRG_TRI_CLUSTER": "0"}, [129, 256, 513]),
])
def test_sectors(env, orders):
    run_child(env, [os.path.join(HERE, "test_gpu_tri_resident.py") + f"::test_sector[{n}]" for n in orders], len(orders))
