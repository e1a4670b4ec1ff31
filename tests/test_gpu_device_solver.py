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


MIXED = """
import math, sys
sys.path[:0] = [{root!r}, {package!r}]
import numpy as np, torch
from nrg_b200 import Context, model, prepare_basis
it, ka, kb = 8, 3500, 100
n = ka + kb
rng = np.random.default_rng(n)
inp = model.siam(U=0.2, Gamma=0.02, eps_d=-0.1, Lambda=2.0, n_keep=64, n_iterations=20)
ctx = Context(0)
ctx.set_model(inp)
rec = np.zeros((n, 5), dtype=np.int32)
rec[:ka, 2], rec[ka:, :2], rec[ka:, 2] = np.arange(1, ka + 1), (1, 1), np.arange(1, kb + 1)
E_old = np.concatenate([np.sort(7 * rng.random(ka)), np.sort(7 * rng.random(kb))])
im = np.zeros((n, n, 2), order="F")
im[:ka, ka:, 0] = rng.standard_normal((ka, kb)) / math.sqrt(n)
bi, si = prepare_basis(inp.operation, 2, rec)
E, V, _, ground = ctx.diagonalization(it, si, bi, E_old, im)
hop = inp.rescaled_chains()[1][it - inp.indexOfFirstIteration, 0]
shift = ground - E[int(si[0, 4]) - 1]
for q in si:
    d, c0, b0 = int(q[2]), int(q[3]) - 1, int(q[4]) - 1
    ref, op = bi[b0:b0 + d, 2] - 1, bi[b0:b0 + d, 4]
    H = np.diag(math.sqrt(inp.Lambda) * E_old[ref])
    for (a, b, t, _), c in zip(inp.coefficient_diagonalization_type, inp.coefficient_diagonalization):
        I, J = np.nonzero(op == a)[0], np.nonzero(op == b)[0]
        B = hop * c * im[np.ix_(ref[J], ref[I], [t - 1])][:, :, 0].T
        H[np.ix_(I, J)], H[np.ix_(J, I)] = B, B.T
    h = torch.from_numpy(H).cuda()
    v = torch.from_numpy(V[c0:c0 + d * d].reshape((d, d), order="F").copy()).cuda()
    e = torch.from_numpy(E[b0:b0 + d] + shift).cuda()
    tol = 20 * d * np.finfo(np.float64).eps
    assert torch.all(torch.diff(e) >= 0)
    assert (v.T @ v - torch.eye(d, dtype=v.dtype, device="cuda")).abs().max() <= tol
    assert (h @ v - v * e).abs().max() <= tol * max(1.0, e.abs().max().item())
    print("order", d)
"""


def test_both_reductions_in_one_group():
    """Sectors beside the streamed reduction's limit (3536), in one size group: 3600 on the multi-kernel
    reduction, 3500 streamed.  Residual and orthogonality as in test_gpu_tri_resident, on the device."""
    root = os.path.dirname(HERE)
    code = MIXED.format(root=root, package=os.path.join(root, "nrg-mpi_b200"))
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, NRG_ENTRY_SOLVER="device"), cwd=root,
                       capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-3000:]
    assert r.stdout.count("order 3600") == 2 and r.stdout.count("order 3500") == 2
